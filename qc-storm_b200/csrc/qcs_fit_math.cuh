// Device arithmetic of the MLEbfgs fit: losses, numerical gradient, BFGS
// update and the fixed iteration schedule, one CUDA thread per ROI.
//
// Bit-level contract: the results equal the reference CUDA kernels' (QC-STORM
// bfgsMLE_dll, compiled by nvcc for sm_100a) bit for bit on the same records.
// The fixed-schedule optimiser with a numerical gradient amplifies any
// rounding difference (one fused multiply-add more or less moves most fits by
// more than 1e-3 px), so matching the reference's results rather than its
// statistics needs the same rounding sequence: every expression keeps the
// reference's operand order and its __expf/__logf intrinsics, and the sums of
// two products, whose fusion nvcc decides from the surrounding code, are
// spelled with explicit round-to-nearest intrinsics chosen per kind and ROI
// size (ArithSpec below).
// References (MLEbfgs/bfgs_MLE_dll x64/bfgsMLE_dll/bfgsMLE_dll/):
//   loss        bfgsMLE_Loc_LD/bfgsMLE_GS2D_core.h:459-518, bfgsMLE_AS3D_core.h:485-544,
//               bfgsMLE_Loc_HD/bfgsMLE_GS2D_2Emitter_core.h:519-592,
//               bfgsMLE_GS2D_3Emitter_core.h:511-589, bfgsMLE_AS3D_2Emitter_core.h:570-644
//   gradient    bfgsMLE_GS2D_core.h:430-454 (same in the other kinds)
//   schedule    bfgsMLE_GS2D_core.h:313-426 (same in the other kinds)
//   BFGS update bfgsMLE_Loc_LD/bfgsMLE_core.h:65-204
#pragma once

#include <cstdint>

namespace qcs {

enum FitKind { kGS2D = 0, kAS3D = 1, k2E = 2, k3E = 3, kAS3D2E = 4 };

// parameters, iterations, loss clamp (0 or 0.01), weighted loss
template <int KIND> struct KindTraits;
template <> struct KindTraits<kGS2D> { enum { P = 5, IT = 8, CLAMP001 = 0, WEIGHTED = 1 }; };
template <> struct KindTraits<kAS3D> { enum { P = 6, IT = 11, CLAMP001 = 1, WEIGHTED = 1 }; };
template <> struct KindTraits<k2E> { enum { P = 8, IT = 13, CLAMP001 = 0, WEIGHTED = 1 }; };
template <> struct KindTraits<k3E> { enum { P = 11, IT = 16, CLAMP001 = 0, WEIGHTED = 0 }; };
template <> struct KindTraits<kAS3D2E> { enum { P = 11, IT = 16, CLAMP001 = 1, WEIGHTED = 0 }; };

constexpr int kBisections = 11;

// Scaled parameterisation: amplitude/128, background/64, 1/(2 sigma^2)/0.1
// (bfgsMLE_core.h:52-60).
#define QCS_ASCALE (128.0f)
#define QCS_BSCALE (64.0f)
#define QCS_SSCALE (0.1f)

// One ROI's pixels as seen by its thread: element k at img[k * ld].
// img holds pairs (photoelectrons max((adu - offset) * gain, 1), its __logf),
// element k at img[k * ld]; w the weighted-MLE mask, element k at w[k * ld].
struct RoiRef {
    const float2 *img;
    const float *w;    // read by the weighted kinds only
    int ld;
};

// Pixel rows are unrolled up to this ROI size; the row loop stays rolled.
// Without the unrolled row a thread's pixel terms form one dependent chain
// (exp -> model -> log -> deviance -> sum) with nothing to overlap it, which
// made 11x11 fits four times slower per pixel than 9x9 ones.  Up to 13 the
// roundings of the loss are fixed in the source (ArithSpec), so unrolling
// changes no result.
constexpr int kUnrollMaxR = 13;

// Contraction of a sum of two products a*b + c*d, the only operand shape
// whose fused multiply-add nvcc chooses from the surrounding code (use
// counts after unrolling) rather than from the expression itself:
//   kFuseFirst   fma(a, b, c*d)     kFuseSecond  fma(c, d, a*b)
//   kNoFuse      a*b + c*d          kCompiler    written as a*b + c*d and
//                                                left to the compiler
enum SumMode { kFuseFirst = 0, kFuseSecond = 1, kNoFuse = 2, kCompiler = 3 };

template <int MODE>
__device__ __forceinline__ float sum_of_products(float a, float b, float c, float d) {
    if (MODE == kFuseFirst) return __fmaf_rn(a, b, __fmul_rn(c, d));
    if (MODE == kFuseSecond) return __fmaf_rn(c, d, __fmul_rn(a, b));
    if (MODE == kNoFuse) return __fadd_rn(__fmul_rn(a, b), __fmul_rn(c, d));
    return a * b + c * d;
}

// Per-kind, per-ROI-size contraction choices of the loss (the squared
// distance of each emitter) and of the weighted-MLE mask exponent.
// SUM2 is the sum of the first two emitters' model terms (multi-emitter kinds).
// The choices below are the ones the reference kernels get from nvcc 12.9 for
// sm_100a, found by running the reference's own kernels on a B200 next to
// each explicit variant of these kernels on the same records and keeping the
// variant whose every output bit matches (tests/test_gpu_reference_parity.py
// re-checks them).  They differ between ROI sizes because nvcc's unrolling,
// and with it the use count that decides each fusion, differs.  Sizes not
// listed keep the plain expression (kCompiler).
// MODEL is amplitude * exp + background of the single-emitter kinds: the
// amplitude product is fused (its only use), the background product is not.
template <int KIND, int R>
struct ArithSpec {
    enum { DIST = kCompiler, MASK = kCompiler, SUM2 = kCompiler };
};
constexpr int kModelSum = kFuseFirst;
template <> struct ArithSpec<kGS2D, 7> { enum { DIST = kFuseFirst, MASK = kNoFuse, SUM2 = kCompiler }; };
template <> struct ArithSpec<kGS2D, 9> { enum { DIST = kFuseSecond, MASK = kCompiler, SUM2 = kCompiler }; };
template <> struct ArithSpec<kGS2D, 11> { enum { DIST = kFuseSecond, MASK = kNoFuse, SUM2 = kCompiler }; };
template <> struct ArithSpec<kGS2D, 13> { enum { DIST = kFuseSecond, MASK = kCompiler, SUM2 = kCompiler }; };
template <> struct ArithSpec<kAS3D, 7> { enum { DIST = kFuseFirst, MASK = kFuseFirst, SUM2 = kCompiler }; };
template <> struct ArithSpec<kAS3D, 9> { enum { DIST = kFuseFirst, MASK = kFuseFirst, SUM2 = kCompiler }; };
template <> struct ArithSpec<kAS3D, 11> { enum { DIST = kFuseFirst, MASK = kFuseFirst, SUM2 = kCompiler }; };
template <> struct ArithSpec<k2E, 7> { enum { DIST = kFuseFirst, MASK = kCompiler, SUM2 = kFuseFirst }; };
template <> struct ArithSpec<k2E, 11> { enum { DIST = kFuseSecond, MASK = kCompiler, SUM2 = kFuseFirst }; };
template <> struct ArithSpec<k3E, 7> { enum { DIST = kFuseSecond, MASK = kCompiler, SUM2 = kFuseFirst }; };
template <> struct ArithSpec<k3E, 11> { enum { DIST = kFuseSecond, MASK = kCompiler, SUM2 = kFuseFirst }; };
template <> struct ArithSpec<kAS3D2E, 7> { enum { DIST = kFuseFirst, MASK = kCompiler, SUM2 = kFuseFirst }; };

// Model exponential of one single-emitter parameter vector v at the pixel
// centred on (cp, rp) (GS2D: v = A, x, y, S, B; AS3D: A, x, y, Sx, Sy, B).
template <int KIND, int DIST>
__device__ __forceinline__ float single_expo(float cp, float rp, const float *v) {
    const float dx = cp - v[1], dy = rp - v[2];
    if (KIND == kGS2D) return __expf(-(sum_of_products<DIST>(dx, dx, dy, dy)) * v[3] * QCS_SSCALE);
    return __expf(-(sum_of_products<DIST>(dx * dx * v[3], QCS_SSCALE, dy * dy * v[4], QCS_SSCALE)));
}

// Poisson deviance term of one pixel given the model exponential e.
template <int KIND>
__device__ __forceinline__ float single_term(float e, const float *v, float pixval, float logpix) {
    const float IVal = sum_of_products<kModelSum>(v[0] * QCS_ASCALE, e, v[KindTraits<KIND>::P - 1], QCS_BSCALE);
    return __fmaf_rn(-pixval, __logf(IVal) - logpix, __fsub_rn(IVal, pixval));
}

template <int R, int KIND, int DIST = ArithSpec<KIND, R>::DIST, int SUM2 = ArithSpec<KIND, R>::SUM2>
__device__ __forceinline__ float loss(const RoiRef &roi, float *Ininf) {
    typedef KindTraits<KIND> T;
#pragma unroll
    for (int k = 0; k < T::P; k++) {
        if (T::CLAMP001) {
            if (Ininf[k] < 0.01f) Ininf[k] = 0.01f;
        } else {
            if (Ininf[k] < 0.0f) Ininf[k] = 0.0f;
        }
    }
    float TotalLoss = 0;
#pragma unroll 1
    for (int row = 0; row < R; row++) {
#pragma unroll(R <= kUnrollMaxR ? R : 1)
        for (int col = 0; col < R; col++) {
            const float2 pl = roi.img[(row * R + col) * roi.ld];
            const float pixval = pl.x, logpix = pl.y;
            const float rowpos = row + 0.5f;
            const float colpos = col + 0.5f;
            float Loss_t;
            if (KIND == kGS2D || KIND == kAS3D) {
                Loss_t = single_term<KIND>(single_expo<KIND, DIST>(colpos, rowpos, Ininf), Ininf, pixval, logpix);
            } else if (KIND == k2E) {
                const float dx0 = colpos - Ininf[1], dy0 = rowpos - Ininf[2];
                const float dx1 = colpos - Ininf[4], dy1 = rowpos - Ininf[5];
                const float A0 = Ininf[0] * QCS_ASCALE, A1 = Ininf[3] * QCS_ASCALE;
                const float e0 = __expf(-(sum_of_products<DIST>(dx0, dx0, dy0, dy0)) * Ininf[6] * QCS_SSCALE);
                const float e1 = __expf(-(sum_of_products<DIST>(dx1, dx1, dy1, dy1)) * Ininf[6] * QCS_SSCALE);
                float IVal_all = sum_of_products<SUM2>(A0, e0, A1, e1) + Ininf[7] * QCS_BSCALE;
                Loss_t = IVal_all - pixval - pixval * (__logf(IVal_all) - logpix);
            } else if (KIND == k3E) {
                const float dx0 = colpos - Ininf[1], dy0 = rowpos - Ininf[2];
                const float dx1 = colpos - Ininf[4], dy1 = rowpos - Ininf[5];
                const float dx2 = colpos - Ininf[7], dy2 = rowpos - Ininf[8];
                const float A0 = Ininf[0] * QCS_ASCALE, A1 = Ininf[3] * QCS_ASCALE, A2 = Ininf[6] * QCS_ASCALE;
                const float e0 = __expf(-(sum_of_products<DIST>(dx0, dx0, dy0, dy0)) * Ininf[9] * QCS_SSCALE);
                const float e1 = __expf(-(sum_of_products<DIST>(dx1, dx1, dy1, dy1)) * Ininf[9] * QCS_SSCALE);
                const float e2 = __expf(-(sum_of_products<DIST>(dx2, dx2, dy2, dy2)) * Ininf[9] * QCS_SSCALE);
                float IVal_all = sum_of_products<SUM2>(A0, e0, A1, e1) + A2 * e2 + Ininf[10] * QCS_BSCALE;
                Loss_t = IVal_all - pixval - pixval * (__logf(IVal_all) - logpix);
            } else {  // kAS3D2E
                const float dx0 = colpos - Ininf[1], dy0 = rowpos - Ininf[2];
                const float dx1 = colpos - Ininf[6], dy1 = rowpos - Ininf[7];
                const float A0 = Ininf[0] * QCS_ASCALE, A1 = Ininf[5] * QCS_ASCALE;
                const float e0 = __expf(-(sum_of_products<DIST>(dx0 * dx0 * Ininf[3], QCS_SSCALE, dy0 * dy0 * Ininf[4],
                                                                QCS_SSCALE)));
                const float e1 = __expf(-(sum_of_products<DIST>(dx1 * dx1 * Ininf[8], QCS_SSCALE, dy1 * dy1 * Ininf[9],
                                                                QCS_SSCALE)));
                float IVal_all = sum_of_products<SUM2>(A0, e0, A1, e1) + Ininf[10] * QCS_BSCALE;
                Loss_t = IVal_all - pixval - pixval * (__logf(IVal_all) - logpix);
            }
            if (T::WEIGHTED)
                TotalLoss = __fmaf_rn(roi.w[(row * R + col) * roi.ld], Loss_t, TotalLoss);
            else
                TotalLoss = __fadd_rn(TotalLoss, Loss_t);
        }
    }
    return TotalLoss;
}

// Central difference on a working copy; each loss call clamps the copy in
// place and later parameters see the clamped values, as in the reference.
template <int R, int KIND, int DIST = ArithSpec<KIND, R>::DIST, int SUM2 = ArithSpec<KIND, R>::SUM2>
__device__ __forceinline__ void numerical_gradient(const RoiRef &roi, const float *Ininf, float *grad) {
    enum { P = KindTraits<KIND>::P };
    float tIninf[P];
#pragma unroll
    for (int cnt = 0; cnt < P; cnt++) tIninf[cnt] = Ininf[cnt];
    for (int cnt = 0; cnt < P; cnt++) {
        tIninf[cnt] = tIninf[cnt] - 0.002f;
        float tgradn = loss<R, KIND, DIST, SUM2>(roi, tIninf);
        tIninf[cnt] = tIninf[cnt] + 0.004f;
        float tgradp = loss<R, KIND, DIST, SUM2>(roi, tIninf);
        grad[cnt] = (tgradp - tgradn) * 250.0f;
        tIninf[cnt] = tIninf[cnt] - 0.002f;
    }
}

// The central-difference gradient of the single-emitter kinds in one sweep
// over the pixels: the 2P evaluation points are first replayed exactly as
// numerical_gradient produces them (with its in-place clamping), then every
// pixel is loaded once and each point's deviance accumulated in its own sum,
// in pixel order.  The amplitude and background points leave the exponent's
// inputs (x, y, widths) unchanged, so their exponential is the base point's;
// this is checked bit for bit per ROI, and a warp with any ROI where it does
// not hold falls back to the point-by-point gradient.  Each sum therefore
// equals the separate loss evaluation bit for bit.
template <int R, int KIND, int DIST = ArithSpec<KIND, R>::DIST>
__device__ __forceinline__ void numerical_gradient_shared(const RoiRef &roi, const float *Ininf, float *grad) {
    typedef KindTraits<KIND> T;
    enum { P = T::P, NE = 2 * P };
    float v[NE][P];
    {
        float t[P];
#pragma unroll
        for (int k = 0; k < P; k++) t[k] = Ininf[k];
#pragma unroll
        for (int k = 0; k < P; k++) {
            t[k] = t[k] - 0.002f;
#pragma unroll
            for (int c = 0; c < P; c++) {
                if (T::CLAMP001) { if (t[c] < 0.01f) t[c] = 0.01f; } else { if (t[c] < 0.0f) t[c] = 0.0f; }
                v[2 * k][c] = t[c];
            }
            t[k] = t[k] + 0.004f;
#pragma unroll
            for (int c = 0; c < P; c++) {
                if (T::CLAMP001) { if (t[c] < 0.01f) t[c] = 0.01f; } else { if (t[c] < 0.0f) t[c] = 0.0f; }
                v[2 * k + 1][c] = t[c];
            }
            t[k] = t[k] - 0.002f;
        }
    }
    bool share = true;
#pragma unroll
    for (int c = 1; c < P - 1; c++) {
        const unsigned b = __float_as_uint(v[0][c]);
        share = share && (__float_as_uint(v[1][c]) == b) && (__float_as_uint(v[NE - 2][c]) == b) &&
                (__float_as_uint(v[NE - 1][c]) == b);
    }
    if (!__all_sync(__activemask(), share)) {
        numerical_gradient<R, KIND, DIST>(roi, Ininf, grad);
        return;
    }
    float tot[NE];
#pragma unroll
    for (int j = 0; j < NE; j++) tot[j] = 0;
#pragma unroll 1
    for (int row = 0; row < R; row++) {
#pragma unroll(R <= kUnrollMaxR ? R : 1)
        for (int col = 0; col < R; col++) {
            const float2 pl = roi.img[(row * R + col) * roi.ld];
            const float pixval = pl.x, logpix = pl.y;
            const float w = T::WEIGHTED ? roi.w[(row * R + col) * roi.ld] : 1.0f;
            const float rowpos = row + 0.5f;
            const float colpos = col + 0.5f;
            const float e_base = single_expo<KIND, DIST>(colpos, rowpos, v[0]);
#pragma unroll
            for (int j = 0; j < NE; j++) {
                const bool base = (j < 2) || (j >= NE - 2);
                const float e = base ? e_base : single_expo<KIND, DIST>(colpos, rowpos, v[j]);
                const float Lt = single_term<KIND>(e, v[j], pixval, logpix);
                tot[j] = T::WEIGHTED ? __fmaf_rn(w, Lt, tot[j]) : __fadd_rn(tot[j], Lt);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < P; k++) grad[k] = (tot[2 * k + 1] - tot[2 * k]) * 250.0f;
}

// D <- (I - s y'/(y's)) D (I - y s'/(y's)) + s s'/(y's); D is row-major P x P
// at D[(r * P + c) * ld].
template <int P>
__device__ __forceinline__ void bfgs_update(float *D, int ld, const float *sk, const float *yk) {
    float divdat = 0;
#pragma unroll
    for (int cnt = 0; cnt < P; cnt++) divdat += sk[cnt] * yk[cnt];
    divdat = 1.0f / divdat;
    float tdat10[P], tdat20[P];
#pragma unroll
    for (int cnt = 0; cnt < P; cnt++) {
        tdat10[cnt] = yk[cnt] * divdat;
        tdat20[cnt] = sk[cnt] * divdat;
    }
    float skyk[P][P], sksk[P][P], tD0[P][P];
#pragma unroll
    for (int row = 0; row < P; row++) {
#pragma unroll
        for (int col = 0; col < P; col++) {
            if (row == col)
                skyk[row][col] = 1.0f - sk[row] * tdat10[col];
            else
                skyk[row][col] = 0.0f - sk[row] * tdat10[col];
            sksk[row][col] = sk[row] * tdat20[col];
        }
    }
#pragma unroll
    for (int row = 0; row < P; row++) {
#pragma unroll
        for (int col = 0; col < P; col++) {
            tD0[row][col] = 0;
#pragma unroll
            for (int cnt = 0; cnt < P; cnt++) tD0[row][col] += skyk[row][cnt] * D[(cnt * P + col) * ld];
        }
    }
#pragma unroll
    for (int row = 0; row < P; row++) {
#pragma unroll
        for (int col = 0; col < P; col++) {
            float acc = 0;
#pragma unroll
            for (int cnt = 0; cnt < P; cnt++) acc += tD0[row][cnt] * skyk[col][cnt];
            D[(row * P + col) * ld] = acc;
        }
    }
#pragma unroll
    for (int row = 0; row < P; row++) {
#pragma unroll
        for (int cnt = 0; cnt < P; cnt++) D[(row * P + cnt) * ld] = D[(row * P + cnt) * ld] + sksk[row][cnt];
    }
}

template <int R, int KIND, int DIST, int SUM2>
__device__ __forceinline__ void gradient(const RoiRef &roi, const float *Ininf, float *grad) {
    if (KIND == kGS2D || KIND == kAS3D)
        numerical_gradient_shared<R, KIND, DIST>(roi, Ininf, grad);
    else
        numerical_gradient<R, KIND, DIST, SUM2>(roi, Ininf, grad);
}

// Loss and gradient of one ROI evaluated by its own thread.
template <int R, int KIND, int DIST, int SUM2>
struct ThreadEval {
    RoiRef roi;
    __device__ __forceinline__ float loss(float *x) const { return qcs::loss<R, KIND, DIST, SUM2>(roi, x); }
    __device__ __forceinline__ void gradient(const float *x, float *g) const {
        qcs::gradient<R, KIND, DIST, SUM2>(roi, x, g);
    }
};

// GS2D loss of ThreadEval with the analytic gradient in one pass over the
// pixels (learned-start fits; the reference's fits use the central
// difference).  With mu = 128 A e + 64 B, e = exp(-0.1 S r^2), r^2 = dx^2 +
// dy^2, dx = col + 0.5 - X, and the weighted deviance sum w (mu - n - n ln
// mu/n), each parameter's derivative is sum w (1 - n / mu) dmu/dtheta:
//   dmu/dA = 128 e, dmu/dX = 128 A e 0.2 S dx, dmu/dY = 128 A e 0.2 S dy,
//   dmu/dS = -128 A e 0.1 r^2, dmu/dB = 64,
// at the point clamped as the loss clamps it.  One exponential and one
// division per pixel instead of the central difference's ten losses.
template <int R, int DIST>
struct AnalyticEvalGS2D {
    RoiRef roi;
    __device__ __forceinline__ float loss(float *x) const {
        return qcs::loss<R, kGS2D, DIST, ArithSpec<kGS2D, R>::SUM2>(roi, x);
    }
    __device__ __forceinline__ void gradient(const float *v, float *g) const {
        float c[5];
#pragma unroll
        for (int k = 0; k < 5; k++) c[k] = v[k] < 0.0f ? 0.0f : v[k];
        const float A128 = c[0] * QCS_ASCALE, B64 = c[4] * QCS_BSCALE, S01 = c[3] * QCS_SSCALE;
        float gA = 0, gX = 0, gY = 0, gS = 0, gB = 0;
#pragma unroll 1
        for (int row = 0; row < R; row++) {
            const float dy = (row + 0.5f) - c[2];
#pragma unroll(R <= kUnrollMaxR ? R : 1)
            for (int col = 0; col < R; col++) {
                const float2 pl = roi.img[(row * R + col) * roi.ld];
                const float w = roi.w[(row * R + col) * roi.ld];
                const float dx = (col + 0.5f) - c[1];
                const float r2 = __fmaf_rn(dx, dx, dy * dy);
                const float e = __expf(-r2 * S01);
                const float mu = __fmaf_rn(A128, e, B64);
                const float q = w * (1.0f - __fdividef(pl.x, mu));
                const float qe = q * e;
                gA += qe;
                gX = __fmaf_rn(qe, dx, gX);
                gY = __fmaf_rn(qe, dy, gY);
                gS = __fmaf_rn(qe, r2, gS);
                gB += q;
            }
        }
        g[0] = QCS_ASCALE * gA;
        g[1] = A128 * 2.0f * S01 * gX;
        g[2] = A128 * 2.0f * S01 * gY;
        g[3] = -A128 * QCS_SSCALE * gS;
        g[4] = QCS_BSCALE * gB;
    }
};

// The same for AS3D (separate widths): with mu = 128 A e + 64 B,
// e = exp(-0.1 (Sx dx^2 + Sy dy^2)),
//   dmu/dA = 128 e, dmu/dX = 128 A e 0.2 Sx dx, dmu/dY = 128 A e 0.2 Sy dy,
//   dmu/dSx = -128 A e 0.1 dx^2, dmu/dSy = -128 A e 0.1 dy^2, dmu/dB = 64,
// at the point clamped as the AS3D loss clamps it (every parameter >= 0.01).
template <int R, int DIST>
struct AnalyticEvalAS3D {
    RoiRef roi;
    __device__ __forceinline__ float loss(float *x) const {
        return qcs::loss<R, kAS3D, DIST, ArithSpec<kAS3D, R>::SUM2>(roi, x);
    }
    __device__ __forceinline__ void gradient(const float *v, float *g) const {
        float c[6];
#pragma unroll
        for (int k = 0; k < 6; k++) c[k] = v[k] < 0.01f ? 0.01f : v[k];
        const float A128 = c[0] * QCS_ASCALE, B64 = c[5] * QCS_BSCALE;
        const float Sx = c[3] * QCS_SSCALE, Sy = c[4] * QCS_SSCALE;
        float gA = 0, gX = 0, gY = 0, gSx = 0, gSy = 0, gB = 0;
#pragma unroll 1
        for (int row = 0; row < R; row++) {
            const float dy = (row + 0.5f) - c[2];
            const float qy = dy * dy;
#pragma unroll(R <= kUnrollMaxR ? R : 1)
            for (int col = 0; col < R; col++) {
                const float2 pl = roi.img[(row * R + col) * roi.ld];
                const float w = roi.w[(row * R + col) * roi.ld];
                const float dx = (col + 0.5f) - c[1];
                const float qx = dx * dx;
                const float e = __expf(-__fmaf_rn(qx, Sx, qy * Sy));
                const float mu = __fmaf_rn(A128, e, B64);
                const float q = w * (1.0f - __fdividef(pl.x, mu));
                const float qe = q * e;
                gA += qe;
                gX = __fmaf_rn(qe, dx, gX);
                gY = __fmaf_rn(qe, dy, gY);
                gSx = __fmaf_rn(qe, qx, gSx);
                gSy = __fmaf_rn(qe, qy, gSy);
                gB += q;
            }
        }
        g[0] = QCS_ASCALE * gA;
        g[1] = A128 * 2.0f * Sx * gX;
        g[2] = A128 * 2.0f * Sy * gY;
        g[3] = -A128 * QCS_SSCALE * gSx;
        g[4] = -A128 * QCS_SSCALE * gSy;
        g[5] = QCS_BSCALE * gB;
    }
};


// The two-emitter GS2D loss (shared S and B, the loss the 2E fit minimises)
// with its analytic gradient: mu = 128 (A0 e0 + A1 e1) + 64 B,
// ek = exp(-0.1 S rk^2), and with q = w (1 - n / mu)
//   dA_k = 128 sum q ek, dX_k = 128 A_k 0.2 S sum q ek dx_k (same for Y),
//   dS = -12.8 sum q (A0 e0 r0^2 + A1 e1 r1^2), dB = 64 sum q,
// at the point clamped as the loss clamps it (parameters >= 0).
template <int R, int DIST>
struct AnalyticEval2E {
    RoiRef roi;
    __device__ __forceinline__ float loss(float *x) const {
        return qcs::loss<R, k2E, DIST, ArithSpec<k2E, R>::SUM2>(roi, x);
    }
    __device__ __forceinline__ void gradient(const float *v, float *g) const {
        float c[8];
#pragma unroll
        for (int k = 0; k < 8; k++) c[k] = v[k] < 0.0f ? 0.0f : v[k];
        const float A0 = c[0] * QCS_ASCALE, A1 = c[3] * QCS_ASCALE, S01 = c[6] * QCS_SSCALE, B64 = c[7] * QCS_BSCALE;
        float gA0 = 0, gX0 = 0, gY0 = 0, gA1 = 0, gX1 = 0, gY1 = 0, gS = 0, gB = 0;
#pragma unroll 1
        for (int row = 0; row < R; row++) {
            const float dy0 = (row + 0.5f) - c[2], dy1 = (row + 0.5f) - c[5];
#pragma unroll(R <= kUnrollMaxR ? R : 1)
            for (int col = 0; col < R; col++) {
                const float2 pl = roi.img[(row * R + col) * roi.ld];
                const float w = roi.w[(row * R + col) * roi.ld];
                const float dx0 = (col + 0.5f) - c[1], dx1 = (col + 0.5f) - c[4];
                const float r0 = __fmaf_rn(dx0, dx0, dy0 * dy0), r1 = __fmaf_rn(dx1, dx1, dy1 * dy1);
                const float e0 = __expf(-r0 * S01), e1 = __expf(-r1 * S01);
                const float mu = __fmaf_rn(A0, e0, __fmaf_rn(A1, e1, B64));
                const float q = w * (1.0f - __fdividef(pl.x, mu));
                const float q0 = q * e0, q1 = q * e1;
                gA0 += q0;
                gX0 = __fmaf_rn(q0, dx0, gX0);
                gY0 = __fmaf_rn(q0, dy0, gY0);
                gA1 += q1;
                gX1 = __fmaf_rn(q1, dx1, gX1);
                gY1 = __fmaf_rn(q1, dy1, gY1);
                gS = __fmaf_rn(A0 * q0, r0, __fmaf_rn(A1 * q1, r1, gS));
                gB += q;
            }
        }
        g[0] = QCS_ASCALE * gA0;
        g[1] = A0 * 2.0f * S01 * gX0;
        g[2] = A0 * 2.0f * S01 * gY0;
        g[3] = QCS_ASCALE * gA1;
        g[4] = A1 * 2.0f * S01 * gX1;
        g[5] = A1 * 2.0f * S01 * gY1;
        g[6] = -QCS_SSCALE * gS;
        g[7] = QCS_BSCALE * gB;
    }
};
// Loss of the GS2D three-emitter fit (the plain kernel's, unweighted) with
// the analytic gradient of that Poisson deviance: d/d mu = 1 - n / mu per
// pixel, chained through the three Gaussians sharing 1/(2 sigma^2) and the
// background (the learned-start three-emitter fit; no central differences).
template <int R, int DIST>
struct AnalyticEval3E {
    RoiRef roi;
    __device__ __forceinline__ float loss(float *x) const {
        return qcs::loss<R, k3E, DIST, ArithSpec<k3E, R>::SUM2>(roi, x);
    }
    __device__ __forceinline__ void gradient(const float *v, float *g) const {
        float c[11];
#pragma unroll
        for (int k = 0; k < 11; k++) c[k] = v[k] < 0.0f ? 0.0f : v[k];
        const float A0 = c[0] * QCS_ASCALE, A1 = c[3] * QCS_ASCALE, A2 = c[6] * QCS_ASCALE;
        const float S = c[9] * QCS_SSCALE, B64 = c[10] * QCS_BSCALE;
        float gA0 = 0, gX0 = 0, gY0 = 0, gA1 = 0, gX1 = 0, gY1 = 0, gA2 = 0, gX2 = 0, gY2 = 0, gS = 0, gB = 0;
#pragma unroll 1
        for (int row = 0; row < R; row++) {
            const float dy0 = (row + 0.5f) - c[2], dy1 = (row + 0.5f) - c[5], dy2 = (row + 0.5f) - c[8];
#pragma unroll(R <= kUnrollMaxR ? R : 1)
            for (int col = 0; col < R; col++) {
                const float2 pl = roi.img[(row * R + col) * roi.ld];
                const float dx0 = (col + 0.5f) - c[1], dx1 = (col + 0.5f) - c[4], dx2 = (col + 0.5f) - c[7];
                const float r0 = __fmaf_rn(dx0, dx0, dy0 * dy0), r1 = __fmaf_rn(dx1, dx1, dy1 * dy1);
                const float r2 = __fmaf_rn(dx2, dx2, dy2 * dy2);
                const float e0 = __expf(-r0 * S), e1 = __expf(-r1 * S), e2 = __expf(-r2 * S);
                const float mu = __fmaf_rn(A0, e0, __fmaf_rn(A1, e1, __fmaf_rn(A2, e2, B64)));
                const float q = 1.0f - __fdividef(pl.x, mu);
                const float q0 = q * e0, q1 = q * e1, q2 = q * e2;
                gA0 += q0;
                gX0 = __fmaf_rn(q0, dx0, gX0);
                gY0 = __fmaf_rn(q0, dy0, gY0);
                gA1 += q1;
                gX1 = __fmaf_rn(q1, dx1, gX1);
                gY1 = __fmaf_rn(q1, dy1, gY1);
                gA2 += q2;
                gX2 = __fmaf_rn(q2, dx2, gX2);
                gY2 = __fmaf_rn(q2, dy2, gY2);
                gS = __fmaf_rn(A0 * q0, r0, __fmaf_rn(A1 * q1, r1, __fmaf_rn(A2 * q2, r2, gS)));
                gB += q;
            }
        }
        g[0] = QCS_ASCALE * gA0;
        g[1] = A0 * 2.0f * S * gX0;
        g[2] = A0 * 2.0f * S * gY0;
        g[3] = QCS_ASCALE * gA1;
        g[4] = A1 * 2.0f * S * gX1;
        g[5] = A1 * 2.0f * S * gY1;
        g[6] = QCS_ASCALE * gA2;
        g[7] = A2 * 2.0f * S * gX2;
        g[8] = A2 * 2.0f * S * gY2;
        g[9] = -QCS_SSCALE * gS;
        g[10] = QCS_BSCALE * gB;
    }
};

// Poisson deviance term of one pixel of the multi-emitter kinds at the
// parameters v: the expressions of loss(), term for term.
template <int KIND, int DIST, int SUM2>
__device__ __forceinline__ float multi_term(float colpos, float rowpos, const float *v, float pixval, float logpix) {
    if (KIND == k2E) {
        const float dx0 = colpos - v[1], dy0 = rowpos - v[2];
        const float dx1 = colpos - v[4], dy1 = rowpos - v[5];
        const float A0 = v[0] * QCS_ASCALE, A1 = v[3] * QCS_ASCALE;
        const float e0 = __expf(-(sum_of_products<DIST>(dx0, dx0, dy0, dy0)) * v[6] * QCS_SSCALE);
        const float e1 = __expf(-(sum_of_products<DIST>(dx1, dx1, dy1, dy1)) * v[6] * QCS_SSCALE);
        float IVal_all = sum_of_products<SUM2>(A0, e0, A1, e1) + v[7] * QCS_BSCALE;
        return IVal_all - pixval - pixval * (__logf(IVal_all) - logpix);
    } else if (KIND == k3E) {
        const float dx0 = colpos - v[1], dy0 = rowpos - v[2];
        const float dx1 = colpos - v[4], dy1 = rowpos - v[5];
        const float dx2 = colpos - v[7], dy2 = rowpos - v[8];
        const float A0 = v[0] * QCS_ASCALE, A1 = v[3] * QCS_ASCALE, A2 = v[6] * QCS_ASCALE;
        const float e0 = __expf(-(sum_of_products<DIST>(dx0, dx0, dy0, dy0)) * v[9] * QCS_SSCALE);
        const float e1 = __expf(-(sum_of_products<DIST>(dx1, dx1, dy1, dy1)) * v[9] * QCS_SSCALE);
        const float e2 = __expf(-(sum_of_products<DIST>(dx2, dx2, dy2, dy2)) * v[9] * QCS_SSCALE);
        float IVal_all = sum_of_products<SUM2>(A0, e0, A1, e1) + A2 * e2 + v[10] * QCS_BSCALE;
        return IVal_all - pixval - pixval * (__logf(IVal_all) - logpix);
    } else {  // kAS3D2E
        const float dx0 = colpos - v[1], dy0 = rowpos - v[2];
        const float dx1 = colpos - v[6], dy1 = rowpos - v[7];
        const float A0 = v[0] * QCS_ASCALE, A1 = v[5] * QCS_ASCALE;
        const float e0 = __expf(-(sum_of_products<DIST>(dx0 * dx0 * v[3], QCS_SSCALE, dy0 * dy0 * v[4], QCS_SSCALE)));
        const float e1 = __expf(-(sum_of_products<DIST>(dx1 * dx1 * v[8], QCS_SSCALE, dy1 * dy1 * v[9], QCS_SSCALE)));
        float IVal_all = sum_of_products<SUM2>(A0, e0, A1, e1) + v[10] * QCS_BSCALE;
        return IVal_all - pixval - pixval * (__logf(IVal_all) - logpix);
    }
}

// The same loss and analytic gradient evaluated by one warp: lane l sums the
// pixels l, l + 32, ...; each sum is reduced by a shuffle tree and lane 0's
// total broadcast, so every lane holds the same value (the lanes' BFGS steps
// stay identical).  img: the ROI's PIX (value, log) pairs, contiguous.
template <int R>
struct AnalyticWarpEval3E {
    const float2 *img;
    int lane;
    unsigned mask;
    __device__ __forceinline__ float uniform_sum(float v) const {
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(mask, v, m);
        return __shfl_sync(mask, v, 0);
    }
    __device__ __forceinline__ float loss(float *x) const {
#pragma unroll
        for (int k = 0; k < 11; k++)
            if (x[k] < 0.0f) x[k] = 0.0f;
        float s = 0.0f;
        for (int k = lane; k < R * R; k += 32) {
            const int row = k / R, col = k - row * R;
            const float2 pl = img[k];
            s += multi_term<k3E, ArithSpec<k3E, R>::DIST, ArithSpec<k3E, R>::SUM2>(col + 0.5f, row + 0.5f, x, pl.x,
                                                                                  pl.y);
        }
        return uniform_sum(s);
    }
    __device__ __forceinline__ void gradient(const float *v, float *g) const {
        float c[11];
#pragma unroll
        for (int k = 0; k < 11; k++) c[k] = v[k] < 0.0f ? 0.0f : v[k];
        const float A[3] = {c[0] * QCS_ASCALE, c[3] * QCS_ASCALE, c[6] * QCS_ASCALE};
        const float S = c[9] * QCS_SSCALE, B64 = c[10] * QCS_BSCALE;
        float gA[3] = {0, 0, 0}, gX[3] = {0, 0, 0}, gY[3] = {0, 0, 0}, gS = 0, gB = 0;
        for (int k = lane; k < R * R; k += 32) {
            const int row = k / R, col = k - row * R;
            const float2 pl = img[k];
            float dx[3], dy[3], r[3], e[3];
#pragma unroll
            for (int j = 0; j < 3; j++) {
                dx[j] = (col + 0.5f) - c[3 * j + 1];
                dy[j] = (row + 0.5f) - c[3 * j + 2];
                r[j] = __fmaf_rn(dx[j], dx[j], dy[j] * dy[j]);
                e[j] = __expf(-r[j] * S);
            }
            const float mu = __fmaf_rn(A[0], e[0], __fmaf_rn(A[1], e[1], __fmaf_rn(A[2], e[2], B64)));
            const float q = 1.0f - __fdividef(pl.x, mu);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const float qj = q * e[j];
                gA[j] += qj;
                gX[j] = __fmaf_rn(qj, dx[j], gX[j]);
                gY[j] = __fmaf_rn(qj, dy[j], gY[j]);
                gS = __fmaf_rn(A[j] * qj, r[j], gS);
            }
            gB += q;
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            g[3 * j] = QCS_ASCALE * uniform_sum(gA[j]);
            g[3 * j + 1] = A[j] * 2.0f * S * uniform_sum(gX[j]);
            g[3 * j + 2] = A[j] * 2.0f * S * uniform_sum(gY[j]);
        }
        g[9] = -QCS_SSCALE * uniform_sum(gS);
        g[10] = QCS_BSCALE * uniform_sum(gB);
    }
};

// Expected photoelectrons of pixel (colpos, rowpos) under the model at the
// parameters v (fit units): the model value of loss(), expression for
// expression.
template <int KIND, int DIST, int SUM2>
__device__ __forceinline__ float model_value(float colpos, float rowpos, const float *v) {
    if (KIND == kGS2D || KIND == kAS3D) {
        const float e = single_expo<KIND, DIST>(colpos, rowpos, v);
        return sum_of_products<kModelSum>(v[0] * QCS_ASCALE, e, v[KindTraits<KIND>::P - 1], QCS_BSCALE);
    } else if (KIND == k2E) {
        const float dx0 = colpos - v[1], dy0 = rowpos - v[2];
        const float dx1 = colpos - v[4], dy1 = rowpos - v[5];
        const float A0 = v[0] * QCS_ASCALE, A1 = v[3] * QCS_ASCALE;
        const float e0 = __expf(-(sum_of_products<DIST>(dx0, dx0, dy0, dy0)) * v[6] * QCS_SSCALE);
        const float e1 = __expf(-(sum_of_products<DIST>(dx1, dx1, dy1, dy1)) * v[6] * QCS_SSCALE);
        return sum_of_products<SUM2>(A0, e0, A1, e1) + v[7] * QCS_BSCALE;
    } else if (KIND == k3E) {
        const float dx0 = colpos - v[1], dy0 = rowpos - v[2];
        const float dx1 = colpos - v[4], dy1 = rowpos - v[5];
        const float dx2 = colpos - v[7], dy2 = rowpos - v[8];
        const float A0 = v[0] * QCS_ASCALE, A1 = v[3] * QCS_ASCALE, A2 = v[6] * QCS_ASCALE;
        const float e0 = __expf(-(sum_of_products<DIST>(dx0, dx0, dy0, dy0)) * v[9] * QCS_SSCALE);
        const float e1 = __expf(-(sum_of_products<DIST>(dx1, dx1, dy1, dy1)) * v[9] * QCS_SSCALE);
        const float e2 = __expf(-(sum_of_products<DIST>(dx2, dx2, dy2, dy2)) * v[9] * QCS_SSCALE);
        return sum_of_products<SUM2>(A0, e0, A1, e1) + A2 * e2 + v[10] * QCS_BSCALE;
    } else {  // kAS3D2E
        const float dx0 = colpos - v[1], dy0 = rowpos - v[2];
        const float dx1 = colpos - v[6], dy1 = rowpos - v[7];
        const float A0 = v[0] * QCS_ASCALE, A1 = v[5] * QCS_ASCALE;
        const float e0 = __expf(-(sum_of_products<DIST>(dx0 * dx0 * v[3], QCS_SSCALE, dy0 * dy0 * v[4], QCS_SSCALE)));
        const float e1 = __expf(-(sum_of_products<DIST>(dx1 * dx1 * v[8], QCS_SSCALE, dy1 * dy1 * v[9], QCS_SSCALE)));
        return sum_of_products<SUM2>(A0, e0, A1, e1) + v[10] * QCS_BSCALE;
    }
}

// Unweighted Poisson log-likelihood of the model at the fitted parameters Ininf
// over pixels k0, k0 + step, ... of the ROI (pixel k's value at img[k]): sum n
// ln(mu) - mu, accumulated in FP64 (the data's ln n! term is common to every
// model of the ROI and left out).  The parameters are clamped as the loss
// clamps them.
template <int R, int KIND, int DIST, int SUM2, class View>
__device__ __forceinline__ double model_loglik(const View &img, const float *Ininf, int k0, int step) {
    typedef KindTraits<KIND> T;
    float v[T::P];
#pragma unroll
    for (int k = 0; k < T::P; k++) v[k] = T::CLAMP001 ? fmaxf(Ininf[k], 0.01f) : fmaxf(Ininf[k], 0.0f);
    double s = 0.0;
    for (int k = k0; k < R * R; k += step) {
        const int row = k / R, col = k - (k / R) * R;
        const double mu = (double)model_value<KIND, DIST, SUM2>(col + 0.5f, row + 0.5f, v);
        s += (double)img[k] * log(mu) - mu;
    }
    return s;
}

// ------------------------------------------------------- packed pairs ---
// Two floats in one 64-bit register pair.  The f32x2 instructions of sm_100
// round each half as the scalar instruction does, at half the issue slots.
// (A packed product whose only use is a packed sum is fused into one
// multiply-add even with .rn on both, so no sum of that shape is written.)
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// (not for a product: see above)
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// e^x = 2^(x log2 e) and ln x = log2(x) ln 2 on the ex2 and lg2 instructions
// that flush subnormals.  Where the result of exp and the argument of log are
// normal the values are those of __expf and __logf bit for bit, and a subnormal
// exp is 0 here (every float is compared in tests/test_gpu_evaluators.py).  They
// take fewer issue slots, which bound the loss with __expf and __logf (85% of the
// slots, 61% of the special-function pipe); the loss takes this form only where
// that changes no sum (flush_safe).
__device__ __forceinline__ float ex2_flush(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 2^x with its subnormal results (and x log2 e for x: __expf of every float).
__device__ __forceinline__ float ex2_keep(float x) {
    float y;
    asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_flush(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ f32x2 ex2_flush2(f32x2 x) {
    float a, b;
    unpack2(x, a, b);
    return pack2(ex2_flush(a), ex2_flush(b));
}
__device__ __forceinline__ f32x2 ex2_keep2(f32x2 x) {
    float a, b;
    unpack2(x, a, b);
    return pack2(ex2_keep(a), ex2_keep(b));
}
__device__ __forceinline__ f32x2 lg2_flush2(f32x2 x) {
    float a, b;
    unpack2(x, a, b);
    return pack2(lg2_flush(a), lg2_flush(b));
}
constexpr float kLog2E = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

// Whether the single-emitter loss at v (already clamped) is the same with the
// flushing forms.  Either the background is large enough that a flushed exp
// (below 2^-126) times the amplitude is under half a unit in the last place
// of every pixel's model value, which then is the background in both forms
// (and a normal number); or (GS2D, whose background may be clamped to zero)
// no pixel's exponent reaches 2^-126 and the amplitude is at least one
// photoelectron, so nothing is subnormal.  The distance of the farthest
// corner bounds every pixel's exponent; 86 leaves its rounding below
// 126 ln 2 = 87.3.  NaN parameters fail both or give NaN in both forms.
template <int R, int KIND>
__device__ __forceinline__ bool flush_safe(const float *v) {
    const float A = v[0] * QCS_ASCALE, B = v[KindTraits<KIND>::P - 1] * QCS_BSCALE;
    bool ok = B >= fmaxf(1e-30f, A * 0x1p-90f);
    if (KIND == kGS2D) {
        const float dx = fmaxf(fabsf(0.5f - v[1]), fabsf((R - 0.5f) - v[1]));
        const float dy = fmaxf(fabsf(0.5f - v[2]), fabsf((R - 0.5f) - v[2]));
        ok = ok || (A >= 1.0f && (dx * dx + dy * dy) * v[3] * QCS_SSCALE <= 86.0f);
    }
    return ok;
}

// ------------------------------------------------------- lane-group fits ---
// Emitters of a kind, and the parameter indices of emitter m's amplitude, x,
// y and widths (Sx = Sy where the kind has one).
template <int KIND>
struct Emitters {
    enum { AS = KIND == kAS3D || KIND == kAS3D2E, M = KIND == k3E ? 3 : ((KIND == k2E || KIND == kAS3D2E) ? 2 : 1) };
    __host__ __device__ static constexpr int a(int m) { return m * (AS ? 5 : 3); }
    __host__ __device__ static constexpr int x(int m) { return a(m) + 1; }
    __host__ __device__ static constexpr int y(int m) { return a(m) + 2; }
    __host__ __device__ static constexpr int sx(int m) { return AS ? a(m) + 3 : KindTraits<KIND>::P - 2; }
    __host__ __device__ static constexpr int sy(int m) { return AS ? a(m) + 4 : KindTraits<KIND>::P - 2; }
    // whether parameter k enters emitter m's exponent
    __host__ __device__ static constexpr bool in(int m, int k) { return k == x(m) || k == y(m) || k == sx(m) || k == sy(m); }
};

// Shared memory of one ROI of a lane group (floats): the pixels' values, then
// their logs, mask (weighted kinds), loss terms [point][pixel], inverse
// Hessian, its update's left product and two parameter vectors.  Pixel rows
// are padded to 4 floats.
template <int R, int KIND>
struct LaneLayout {
    enum {
        P = KindTraits<KIND>::P,
        PIX = R * R,
        PIXP = (PIX + 3) / 4 * 4,
        VAL = 0,
        LOG = VAL + PIXP,
        W = LOG + PIXP,
        PART = W + (KindTraits<KIND>::WEIGHTED ? PIXP : 0),
        H = PART + 2 * P * PIXP,
        T = H + P * P,
        VEC = T + P * P,
        TOTAL = (VEC + 2 * P + 3) / 4 * 4,
    };
};

// One ROI's fit by a group of G consecutive lanes of a warp, the rows of the
// one-thread kernels bit for bit: every term, every sum's order and every
// rounding is theirs; the lanes only divide the work.
//  - Line search: the next midpoint and the one after it do not depend on the
//    comparison between them, and the third has two candidates, so one round
//    evaluates three steps: 4 points on G / 4 lanes each (first the ends and
//    the first midpoint), then the lanes 0..3 sum one point's terms each, in
//    pixel order.  The 12 evaluations one after the other take 4 rounds.
//  - Gradient: a lane computes its pixels' terms at all 2P difference points,
//    each distinct exponential once (a parameter's two points differ only in
//    that parameter, and after it is moved back its rounded value stays: 26
//    exponentials instead of 66 for three emitters), then lane j sums point j.
//  - The inverse Hessian's update: one element per lane and round.
// A line-search term takes two pixels at a time in packed instructions, with the
// flushing exp and log where safe() and, for several emitters, exps_normal() say
// that they change nothing.  The latter is asked once a line search, and point by
// point only where the line as a whole fails it: 2E, 3E and 1E stages of 100,000
// 11x11 records 2,083 -> 2,095 us with it (2,119 with the keeping exp throughout,
// 2,106 with the general terms where a point fails).
// Only for roundings fixed in the source (DIST, SUM2 != kCompiler).  pos: the
// pixels' centres, col + 0.5 of PIXP pixels, then row + 0.5.
template <int R, int KIND, int DIST, int G>
struct LaneFit {
    typedef KindTraits<KIND> T;
    typedef Emitters<KIND> E;
    typedef LaneLayout<R, KIND> L;
    enum { P = T::P, NE = 2 * P, PIX = R * R, PIXP = L::PIXP, KPTS = 4, LP = G / KPTS, LOW = T::CLAMP001 };
    const float *pos;
    float *s;  // the ROI's LaneLayout
    int lane;
    unsigned mask;

    __device__ __forceinline__ static float bound(float v) {
        if (LOW) return v < 0.01f ? 0.01f : v;
        return v < 0.0f ? 0.0f : v;
    }
    // Whether the flushing log, and for one emitter the flushing exp, change
    // nothing at clamped parameters with this background and amplitude: the
    // model is then at least the background, a normal number, and an exp below
    // 2^-126 times the amplitude is lost under it (flush_safe).
    __device__ __forceinline__ static bool safe(float B, float A) {
        return B * QCS_BSCALE >= (E::M == 1 ? fmaxf(1e-30f, A * QCS_ASCALE * 0x1p-45f) : 1e-30f);
    }
    // Whether no exp is subnormal at any (clamped) parameters between v and u and
    // 0.01 beyond, so that the flushing exp is the other's value.  With several
    // emitters the background's size does not settle that: where one emitter's
    // product is a tie of the model's sum, another's subnormal exp decides the
    // rounding.  The farthest pixel and the widest spread bound every exponent;
    // 86 leaves its rounding below 126 ln 2 = 87.3.  A NaN parameter is NaN in
    // both forms.
    __device__ __forceinline__ static bool exps_normal(const float (&v)[P], const float (&u)[P]) {
        if (E::M == 1) return true;  // safe() is enough
        float dx = 0.0f, dy = 0.0f, sx = 0.0f, sy = 0.0f;
#pragma unroll
        for (int m = 0; m < E::M; m++) {
            dx = fmaxf(dx, fmaxf(fabsf(v[E::x(m)] - R / 2.0f), fabsf(u[E::x(m)] - R / 2.0f)));
            dy = fmaxf(dy, fmaxf(fabsf(v[E::y(m)] - R / 2.0f), fabsf(u[E::y(m)] - R / 2.0f)));
            sx = fmaxf(sx, fmaxf(v[E::sx(m)], u[E::sx(m)]));
            sy = fmaxf(sy, fmaxf(v[E::sy(m)], u[E::sy(m)]));
        }
        dx += R / 2 + 0.01f;
        dy += R / 2 + 0.01f;
        return (dx * dx * (sx + 0.01f) + dy * dy * (sy + 0.01f)) * QCS_SSCALE <= 86.0f;
    }
    __device__ __forceinline__ static float exponent(float cp, float rp, float x, float y, float sx, float sy) {
        const float dx = cp - x, dy = rp - y;
        if (E::AS) return -sum_of_products<DIST>(__fmul_rn(__fmul_rn(dx, dx), sx), QCS_SSCALE,
                                                 __fmul_rn(__fmul_rn(dy, dy), sy), QCS_SSCALE);
        return __fmul_rn(__fmul_rn(-sum_of_products<DIST>(dx, dx, dy, dy), sx), QCS_SSCALE);
    }
    template <bool KEEP>
    __device__ __forceinline__ static float expo(float cp, float rp, float x, float y, float sx, float sy) {
        const float t = __fmul_rn(exponent(cp, rp, x, y, sx, sy), kLog2E);
        return KEEP ? ex2_keep(t) : ex2_flush(t);
    }
    // deviance term from the emitters' exponentials e and amplitudes A, and the background B (fit units)
    __device__ __forceinline__ static float term(const float (&e)[E::M], const float (&A)[E::M], float B, float2 pl) {
        float I;
        if (E::M == 1) {
            I = __fmaf_rn(A[0] * QCS_ASCALE, e[0], B * QCS_BSCALE);
        } else {
            I = __fmaf_rn(A[0] * QCS_ASCALE, e[0], __fmul_rn(A[E::M > 1 ? 1 : 0] * QCS_ASCALE, e[E::M > 1 ? 1 : 0]));
            if (E::M > 2) I = __fmaf_rn(A[E::M - 1] * QCS_ASCALE, e[E::M - 1], I);
            I = __fadd_rn(I, B * QCS_BSCALE);
        }
        return __fmaf_rn(pl.x, __fmaf_rn(lg2_flush(I), -kLn2, pl.y), __fsub_rn(I, pl.x));
    }
    // pixel k's term as the one-thread kernels form it, with __expf and __logf
    __device__ __forceinline__ float term_general(int k, const float *v) const {
        const float cp = pos[k], rp = pos[PIXP + k], pix = s[L::VAL + k], lg = s[L::LOG + k];
        if constexpr (E::M == 1)
            return single_term<KIND>(single_expo<KIND, DIST>(cp, rp, v), v, pix, lg);
        else
            return multi_term<KIND, DIST, kFuseFirst>(cp, rp, v, pix, lg);
    }
    __device__ __forceinline__ static f32x2 pair_at(const float *p) { return *reinterpret_cast<const f32x2 *>(p); }
    // expo and term of two pixels
    template <bool KEEP>
    __device__ __forceinline__ static f32x2 expo2(f32x2 cp, f32x2 rp, f32x2 x, f32x2 y, f32x2 sx, f32x2 sy) {
        const f32x2 s01 = pack2(QCS_SSCALE, QCS_SSCALE), dx = sub2(cp, x), dy = sub2(rp, y);
        f32x2 t;
        if (E::AS) {
            t = mul2(fma2(mul2(mul2(dx, dx), sx), s01, mul2(mul2(mul2(dy, dy), sy), s01)), pack2(-kLog2E, -kLog2E));
        } else {
            // -d S: sx is -S
            const f32x2 d = DIST == kFuseFirst ? fma2(dx, dx, mul2(dy, dy)) : fma2(dy, dy, mul2(dx, dx));
            t = mul2(mul2(mul2(d, sx), s01), pack2(kLog2E, kLog2E));
        }
        return KEEP ? ex2_keep2(t) : ex2_flush2(t);
    }
    __device__ __forceinline__ static f32x2 term2(const f32x2 (&e)[E::M], const f32x2 (&A)[E::M], f32x2 B, f32x2 pix,
                                                  f32x2 lg) {
        f32x2 I;
        if (E::M == 1) {
            I = fma2(A[0], e[0], B);
        } else {
            I = fma2(A[0], e[0], mul2(A[E::M > 1 ? 1 : 0], e[E::M > 1 ? 1 : 0]));
            if (E::M > 2) I = fma2(A[E::M - 1], e[E::M - 1], I);
            I = add2(I, B);
        }
        return fma2(pix, fma2(lg2_flush2(I), pack2(-kLn2, -kLn2), lg), sub2(I, pix));
    }

    // Sum of term row j (PIX terms in pixel order, with the mask where the kind is weighted).
    __device__ __forceinline__ float row_sum(int j) const {
        const float4 *p4 = reinterpret_cast<const float4 *>(s + L::PART + j * PIXP);
        const float4 *w4 = reinterpret_cast<const float4 *>(s + L::W);
        float total = 0.0f;
#pragma unroll(PIX <= 49 ? PIX / 4 : 8)
        for (int q = 0; q < PIX / 4; q++) {
            const float4 t = p4[q];
            if (T::WEIGHTED) {
                const float4 a = w4[q];
                total = __fmaf_rn(a.x, t.x, total);
                total = __fmaf_rn(a.y, t.y, total);
                total = __fmaf_rn(a.z, t.z, total);
                total = __fmaf_rn(a.w, t.w, total);
            } else {
                total = __fadd_rn(total, t.x);
                total = __fadd_rn(total, t.y);
                total = __fadd_rn(total, t.z);
                total = __fadd_rn(total, t.w);
            }
        }
#pragma unroll
        for (int k = PIX / 4 * 4; k < PIX; k++) {
            const float t = s[L::PART + j * PIXP + k];
            total = T::WEIGHTED ? __fmaf_rn(s[L::W + k], t, total) : __fadd_rn(total, t);
        }
        return total;
    }

    // The terms of pixels 2 k0, 2 k0 + 1, 2 (k0 + LP), ... at v into part, two at a time.
    template <bool KEEP>
    __device__ __forceinline__ void terms(const float (&v)[P], float *part, int k0) const {
        f32x2 A2[E::M], x2[E::M], y2[E::M], sx2[E::M], sy2[E::M];
        const f32x2 B2 = pack2(v[P - 1] * QCS_BSCALE, v[P - 1] * QCS_BSCALE);
#pragma unroll
        for (int m = 0; m < E::M; m++) {
            const float A = v[E::a(m)] * QCS_ASCALE, sx = E::AS ? v[E::sx(m)] : -v[E::sx(m)], sy = v[E::sy(m)];
            A2[m] = pack2(A, A);
            x2[m] = pack2(v[E::x(m)], v[E::x(m)]);
            y2[m] = pack2(v[E::y(m)], v[E::y(m)]);
            sx2[m] = pack2(sx, sx);
            sy2[m] = pack2(sy, sy);
        }
// (unrolled rounds are slower: the loop is short and the kernel is bound by instruction fetch as well)
#pragma unroll 1
        for (int k = 2 * k0; k < PIX; k += 2 * LP) {
            const f32x2 cp = pair_at(pos + k), rp = pair_at(pos + PIXP + k);
            f32x2 e[E::M];
#pragma unroll
            for (int m = 0; m < E::M; m++) e[m] = expo2<KEEP>(cp, rp, x2[m], y2[m], sx2[m], sy2[m]);
            *reinterpret_cast<f32x2 *>(part + k) = term2(e, A2, B2, pair_at(s + L::VAL + k), pair_at(s + L::LOG + k));
        }
    }

    // Losses at x + d * step[j], j < KPTS, in every lane; normal: exps_normal
    // holds there.
    __device__ __forceinline__ void losses(const float *x, const float *d, const float (&step)[KPTS], bool normal,
                                           float (&f)[KPTS]) const {
        const int j = lane / LP, k0 = lane - j * LP;
        float st = step[0];
#pragma unroll
        for (int i = 1; i < KPTS; i++) st = j == i ? step[i] : st;
        float v[P];
#pragma unroll
        for (int k = 0; k < P; k++) v[k] = bound(__fmaf_rn(d[k], st, x[k]));
        float *part = s + L::PART + j * PIXP;
        if (__all_sync(mask, safe(v[P - 1], v[0]))) {
            if (normal || __all_sync(mask, exps_normal(v, v)))
                terms<false>(v, part, k0);
            else
                terms<true>(v, part, k0);
        } else {
#pragma unroll 1
            for (int k = k0; k < PIX; k += LP) part[k] = term_general(k, v);
        }
        __syncwarp(mask);
        const float total = row_sum(lane & (KPTS - 1));
#pragma unroll
        for (int i = 0; i < KPTS; i++) f[i] = __shfl_sync(mask, total, i, G);
        __syncwarp(mask);
    }

    // The terms of this lane's pixels at the gradient's 2P points into part (see gradient).
    template <bool KEEP>
    __device__ __forceinline__ void point_terms(const float (&b)[P], const float (&lo)[P], const float (&hi)[P],
                                                const float (&r)[P], float *part) const {
#pragma unroll 1
        for (int k = lane; k < PIX; k += G) {
            const float2 c = make_float2(pos[k], pos[PIXP + k]), pl = make_float2(s[L::VAL + k], s[L::LOG + k]);
            float v[P], e[E::M];
#pragma unroll
            for (int i = 0; i < P; i++) v[i] = b[i];
#pragma unroll
            for (int m = 0; m < E::M; m++) e[m] = 0.0f;
#pragma unroll
            for (int i = 0; i < P; i++) {
                float A[E::M], en[E::M];
                // emitters whose exponent the parameter before this one moved, or none is known yet
#pragma unroll
                for (int m = 0; m < E::M; m++)
                    if (!E::in(m, i) && (i == 0 || E::in(m, i - 1)))
                        e[m] = expo<KEEP>(c.x, c.y, v[E::x(m)], v[E::y(m)], v[E::sx(m)], v[E::sy(m)]);
#pragma unroll
                for (int side = 0; side < 2; side++) {
                    v[i] = side ? hi[i] : lo[i];
#pragma unroll
                    for (int m = 0; m < E::M; m++) {
                        A[m] = v[E::a(m)];
                        en[m] = E::in(m, i) ? expo<KEEP>(c.x, c.y, v[E::x(m)], v[E::y(m)], v[E::sx(m)], v[E::sy(m)]) : e[m];
                    }
                    part[(2 * i + side) * PIXP + k] = term(en, A, v[P - 1], pl);
                }
                v[i] = r[i];
            }
        }
    }

    // (normal: exps_normal holds at x)
    __device__ __forceinline__ void gradient(const float *x, float *grad, bool normal) const {
        // parameter k: b before it is moved, lo / hi its two points, r after it is moved back
        float b[P], lo[P], hi[P], r[P];
#pragma unroll
        for (int k = 0; k < P; k++) {
            // (the first loss call, at parameter 0's lower point, clamps all the others)
            b[k] = bound(x[k]);
            lo[k] = bound((k == 0 ? x[k] : b[k]) - 0.002f);
            hi[k] = bound(lo[k] + 0.004f);
            r[k] = bound(hi[k] - 0.002f);
        }
        float *part = s + L::PART;
        const float A = fmaxf(b[0], fmaxf(hi[0], r[0]));
        if (safe(lo[P - 1], A) && safe(b[P - 1], A)) {
            if (normal || exps_normal(b, b))  // (every point is within 0.0041 of b)
                point_terms<false>(b, lo, hi, r, part);
            else
                point_terms<true>(b, lo, hi, r, part);
        } else {
#pragma unroll 1
            for (int j = 0; j < NE; j++) {
                float v[P];
#pragma unroll
                for (int i = 0; i < P; i++) v[i] = i == j / 2 ? ((j & 1) ? hi[i] : lo[i]) : (i < j / 2 ? r[i] : b[i]);
#pragma unroll 1
                for (int k = lane; k < PIX; k += G) part[j * PIXP + k] = term_general(k, v);
            }
        }
        __syncwarp(mask);
        enum { PASSES = (NE + G - 1) / G };
        float tot[PASSES];
#pragma unroll
        for (int p = 0; p < PASSES; p++) tot[p] = row_sum(min(lane + p * G, NE - 1));
#pragma unroll
        for (int k = 0; k < P; k++) {
            const float tn = __shfl_sync(mask, tot[(2 * k) / G], (2 * k) % G, G);
            const float tp = __shfl_sync(mask, tot[(2 * k + 1) / G], (2 * k + 1) % G, G);
            grad[k] = (tp - tn) * 250.0f;
        }
        __syncwarp(mask);
    }

    // bfgs_update and the new direction -D grad, operation for operation (its
    // temporaries recomputed with the roundings nvcc gives their expressions:
    // one fused multiply-add or separate product each, the final s s'/(y's)
    // fused into the sum).
    __device__ __forceinline__ void update(const float *sk, const float *yk, const float *grad, float *d) const {
        float *D = s + L::H, *Tm = s + L::T, *vec = s + L::VEC;
        float divdat = 0.0f;
#pragma unroll
        for (int c = 0; c < P; c++) divdat = __fmaf_rn(sk[c], yk[c], divdat);
        divdat = 1.0f / divdat;
        float t10[P];
#pragma unroll
        for (int c = 0; c < P; c++) t10[c] = __fmul_rn(yk[c], divdat);
        if (lane == 0) {
#pragma unroll
            for (int c = 0; c < P; c++) {
                vec[c] = sk[c];
                vec[P + c] = __fmul_rn(sk[c], divdat);
            }
        }
        __syncwarp(mask);
#pragma unroll 1
        for (int e = lane; e < P * P; e += G) {
            const int row = e / P, col = e - (e / P) * P;
            const float sr = -vec[row];
            float acc = 0.0f;
#pragma unroll
            for (int c = 0; c < P; c++) acc = __fmaf_rn(__fmaf_rn(sr, t10[c], row == c ? 1.0f : 0.0f), D[c * P + col], acc);
            Tm[e] = acc;
        }
        __syncwarp(mask);
#pragma unroll 1
        for (int e = lane; e < P * P; e += G) {
            const int row = e / P, col = e - (e / P) * P;
            const float sc = -vec[col];
            float acc = 0.0f;
#pragma unroll
            for (int c = 0; c < P; c++) acc = __fmaf_rn(Tm[row * P + c], __fmaf_rn(sc, t10[c], col == c ? 1.0f : 0.0f), acc);
            D[e] = __fmaf_rn(vec[row], vec[P + col], acc);
        }
        __syncwarp(mask);
        const int row = min(lane, P - 1);
        float acc = 0.0f;
#pragma unroll
        for (int c = 0; c < P; c++) acc = __fmaf_rn(-D[row * P + c], grad[c], acc);
#pragma unroll
        for (int c = 0; c < P; c++) d[c] = __shfl_sync(mask, acc, c, G);
    }

    // bfgs_fit's schedule
    __device__ __forceinline__ void fit(float *x) const {
        static_assert(kBisections == 11 && P <= G, "one evaluation, then three rounds of three; one direction per lane");
        float grad[P], d[P];
        for (int e = lane; e < P * P; e += G) s[L::H + e] = e % (P + 1) == 0 ? 1.0f : 0.0f;
        gradient(x, grad, false);
#pragma unroll
        for (int k = 0; k < P; k++) d[k] = -grad[k];
#pragma unroll 1
        for (int it = 0; it < T::IT; it++) {
            float total = 0.0f;
#pragma unroll
            for (int k = 0; k < P; k++) total += fabsf(d[k]);
            total = ((float)P) / total;
#pragma unroll
            for (int k = 0; k < P; k++) d[k] = d[k] * total;
            bool normal;  // along the whole line
            {
                float v[P], u[P];
#pragma unroll
                for (int k = 0; k < P; k++) {
                    v[k] = x[k];
                    u[k] = x[k] + d[k];
                }
                normal = exps_normal(v, u);
            }
            float p0 = 0.00001f, p1 = 1.0f, f0 = 0.0f, f1 = 0.0f, f[KPTS];
            // one bisection step: the moved end takes the midpoint and its loss
            auto move = [&](float fm) {
                const bool down = f0 < f1;
                const float mid = (p0 + p1) * 0.5f;
                p0 = down ? p0 : mid;
                p1 = down ? mid : p1;
                f0 = down ? f0 : fm;
                f1 = down ? fm : f1;
            };
            {
                const float st[KPTS] = {0.0001f, 1.0f, (p0 + p1) * 0.5f, 0.0001f};
                losses(x, d, st, normal, f);
                f0 = f[0];
                f1 = f[1];
                move(f[2]);
            }
#pragma unroll 1
            for (int round = 0; round < 3; round++) {
                const bool down = f0 < f1;
                const float m1 = (p0 + p1) * 0.5f;
                const float q0 = down ? p0 : m1, q1 = down ? m1 : p1;
                const float m2 = (q0 + q1) * 0.5f;
                // the third midpoint: the lower half kept (upper end moved to m2), or the upper
                const float st[KPTS] = {m1, m2, (q0 + m2) * 0.5f, (m2 + q1) * 0.5f};
                losses(x, d, st, normal, f);
                move(f[0]);
                const bool lower = f0 < f1;
                move(f[1]);
                move(lower ? f[2] : f[3]);
            }
            const bool down = f0 < f1;  // the last step moves an end without an evaluation
            const float mid = (p0 + p1) * 0.5f;
            p0 = down ? p0 : mid;
            p1 = down ? mid : p1;
            const float scale = (p0 + p1) * 0.5f;
            float sk[P];
#pragma unroll
            for (int k = 0; k < P; k++) {
                sk[k] = d[k] * scale;
                x[k] = x[k] + sk[k];
            }
#pragma unroll
            for (int k = 0; k < P; k++)
                if (x[k] < 0.01f) x[k] = 0.01f;
            if (it < T::IT - 1) {
                float yk[P];
#pragma unroll
                for (int k = 0; k < P; k++) yk[k] = grad[k];
                gradient(x, grad, normal);  // x is on the line, or raised to 0.01
#pragma unroll
                for (int k = 0; k < P; k++) yk[k] = grad[k] - yk[k];
                update(sk, yk, grad, d);
            }
        }
    }
};

// ------------------------------------------ staged single-emitter eval ---
// The weighted-MLE mask of an R x R ROI depends on |col - R/2| and
// |row - R/2| only: its exponent holds the squared distances of the pixel
// centre from the ROI centre, which are equal (exact small numbers) for
// mirrored pixels.  A thread therefore keeps U x U values (U = R/2 + 1);
// mask row ur is C4 float4 chunks, value (ur, uc) in chunk uc / 4, lane uc % 4.
// That holds where the mask's contraction is fixed in the source (MASK !=
// kCompiler).  Where nvcc chooses it, its choice differs between pixels (and
// with the surrounding code), so mirrored pixels need not agree bit for bit:
// there (FULL) the whole R x R mask of wle_weights is kept, pixel k at
// k * ld floats, which reproduces the reference's values.
template <int R, bool FULL = false>
struct MaskShape {
    enum { U = R / 2 + 1, C4 = (U + 3) / 4, FLOATS = FULL ? R * R : U * C4 * 4 };
};

__host__ __device__ constexpr int mirror_index(int k, int R) { return k < R / 2 ? R / 2 - k : k - R / 2; }

// wle_weights for the pixels col, row >= R/2 (same expressions, so the same
// values as at their mirror images), chunk c of mask row ur at wu[(ur * C4 + c) * ld].
template <int R, int MASK = kCompiler>
__device__ __forceinline__ void wle_weights_unique(float4 *wu, int ld, float WLE_SigmaX, float WLE_SigmaY,
                                                   int MoleculeType) {
    typedef MaskShape<R> M;
    const float ROICenter = R / 2.0f;
    const float WLE_SigmaX1 = 1.0f / (2.0f * WLE_SigmaX * WLE_SigmaX);
    const float WLE_SigmaY1 = 1.0f / (2.0f * WLE_SigmaY * WLE_SigmaY);
    for (int ur = 0; ur < M::U; ur++) {
        const float rowpos = (R / 2 + ur) + 0.5f;
        for (int c = 0; c < M::C4; c++) {
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int uc = c * 4 + j;
                const float colpos = (R / 2 + uc) + 0.5f;
                if (MoleculeType == 0 || uc >= M::U)
                    v[j] = 1.0f;
                else
                    v[j] = __expf(-sum_of_products<MASK>((colpos - ROICenter) * (colpos - ROICenter), WLE_SigmaX1,
                                                         (rowpos - ROICenter) * (rowpos - ROICenter), WLE_SigmaY1));
            }
            wu[(ur * M::C4 + c) * ld] = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

// Model exponential of single_expo from the pixel's offsets dx = col + 0.5 - x
// and dy = row + 0.5 - y (the same roundings).
template <int KIND, int DIST>
__device__ __forceinline__ float single_expo_d(float dx, float dy, const float *v) {
    if (KIND == kGS2D) return __expf(-(sum_of_products<DIST>(dx, dx, dy, dy)) * v[3] * QCS_SSCALE);
    return __expf(-(sum_of_products<DIST>(dx * dx * v[3], QCS_SSCALE, dy * dy * v[4], QCS_SSCALE)));
}

// A thread's weighted-MLE mask (MaskShape): unique values as float4 chunks at
// ((const float4 *)mask)[(ur * C4 + c) * ld] (16-byte aligned), or (FULL) the
// R x R values, pixel k at mask[k * ld].
template <int R, bool FULL>
struct MaskView {
    typedef MaskShape<R> M;
    const float *mask;
    int ld;

    // the mask values of `row`, indexed by wcol(col)
    __device__ __forceinline__ void mask_row(int row, float (&w)[FULL ? R : M::C4 * 4]) const {
        if constexpr (FULL) {
#pragma unroll
            for (int c = 0; c < R; c++) w[c] = mask[(row * R + c) * ld];
        } else {
            const int ur = mirror_index(row, R);
            const float4 *wu = reinterpret_cast<const float4 *>(mask);
#pragma unroll
            for (int c = 0; c < M::C4; c++) {
                const float4 q = wu[(ur * M::C4 + c) * ld];
                w[4 * c] = q.x;
                w[4 * c + 1] = q.y;
                w[4 * c + 2] = q.z;
                w[4 * c + 3] = q.w;
            }
        }
    }
    __device__ __forceinline__ static constexpr int wcol(int col) { return FULL ? col : mirror_index(col, R); }
    __device__ __forceinline__ float mask_at(int row, int col) const {
        if constexpr (FULL) return mask[(row * R + col) * ld];
        const int ur = mirror_index(row, R), uc = mirror_index(col, R);
        return mask[((ur * M::C4 + uc / 4) * ld) * 4 + uc % 4];
    }
};

// The 2P central-difference points of the gradient at Ininf, as
// numerical_gradient produces them (each loss call clamps its point in place
// and the next point starts from the clamped values): v[2k] and v[2k + 1] are
// parameter k's lower and upper point.  Returns whether the amplitude and
// background points share the first point's exponent inputs bit for bit.
template <int KIND>
__device__ __forceinline__ bool gradient_points(const float *Ininf, float (&v)[2 * KindTraits<KIND>::P][KindTraits<KIND>::P]) {
    typedef KindTraits<KIND> T;
    enum { P = T::P, NE = 2 * P };
    float t[P];
#pragma unroll
    for (int k = 0; k < P; k++) t[k] = Ininf[k];
#pragma unroll
    for (int k = 0; k < P; k++) {
        t[k] = t[k] - 0.002f;
#pragma unroll
        for (int c = 0; c < P; c++) {
            if (T::CLAMP001) { if (t[c] < 0.01f) t[c] = 0.01f; } else { if (t[c] < 0.0f) t[c] = 0.0f; }
            v[2 * k][c] = t[c];
        }
        t[k] = t[k] + 0.004f;
#pragma unroll
        for (int c = 0; c < P; c++) {
            if (T::CLAMP001) { if (t[c] < 0.01f) t[c] = 0.01f; } else { if (t[c] < 0.0f) t[c] = 0.0f; }
            v[2 * k + 1][c] = t[c];
        }
        t[k] = t[k] - 0.002f;
    }
    bool share = true;
#pragma unroll
    for (int c = 1; c < P - 1; c++) {
        const unsigned b = __float_as_uint(v[0][c]);
        share = share && (__float_as_uint(v[1][c]) == b) && (__float_as_uint(v[NE - 2][c]) == b) &&
                (__float_as_uint(v[NE - 1][c]) == b);
    }
    return share;
}

// Loss and gradient of one single-emitter ROI (GS2D / AS3D) evaluated by its
// own thread, with the pixels' (value, log) pairs at img[k * ld] and the mask
// of MaskView.  Same terms, same order, same roundings as loss() /
// numerical_gradient_shared(), with fewer instructions: one 16-byte mask load
// per row, the column offsets of the position computed once per evaluation,
// the row centre kept as a float.  For the sizes whose distance rounding is
// nvcc's (kCompiler); the others take PairEval.
template <int R, int KIND, int DIST, bool FULL = false>
struct StagedEval : MaskView<R, FULL> {
    typedef KindTraits<KIND> T;
    typedef MaskShape<R> M;
    typedef MaskView<R, FULL> V;
    using V::ld;
    using V::mask_at;
    using V::mask_row;
    using V::wcol;
    enum { P = T::P, UNROLL = R <= kUnrollMaxR };
    const float2 *img;
    __device__ __forceinline__ StagedEval(const float *pix, const float *mask_, int slot, int ld_)
        : V{mask_, ld_}, img(reinterpret_cast<const float2 *>(pix) + slot) {}
    __device__ __forceinline__ float2 pixel(int row, int col) const { return img[(row * R + col) * ld]; }

    __device__ __forceinline__ float loss(float *Ininf) const {
#pragma unroll
        for (int k = 0; k < P; k++) {
            if (T::CLAMP001) {
                if (Ininf[k] < 0.01f) Ininf[k] = 0.01f;
            } else {
                if (Ininf[k] < 0.0f) Ininf[k] = 0.0f;
            }
        }
        float TotalLoss = 0;
        if constexpr (UNROLL) {
            float dxs[R];
#pragma unroll
            for (int col = 0; col < R; col++) dxs[col] = (col + 0.5f) - Ininf[1];
            float rowpos = 0.5f;
            const float2 *pr = img;
#pragma unroll 1
            for (int row = 0; row < R; row++) {
                float w[FULL ? R : M::C4 * 4];
                mask_row(row, w);
                const float dy = rowpos - Ininf[2];
#pragma unroll
                for (int col = 0; col < R; col++) {
                    const float2 pl = pr[col * ld];
                    const float Lt = single_term<KIND>(single_expo_d<KIND, DIST>(dxs[col], dy, Ininf), Ininf, pl.x,
                                                       pl.y);
                    TotalLoss = __fmaf_rn(w[wcol(col)], Lt, TotalLoss);
                }
                rowpos += 1.0f;
                pr += R * ld;
            }
        } else {
#pragma unroll 1
            for (int row = 0; row < R; row++) {
#pragma unroll 1
                for (int col = 0; col < R; col++) {
                    const float2 pl = img[(row * R + col) * ld];
                    const float Lt = single_term<KIND>(
                        single_expo<KIND, DIST>(col + 0.5f, row + 0.5f, Ininf), Ininf, pl.x, pl.y);
                    TotalLoss = __fmaf_rn(mask_at(row, col), Lt, TotalLoss);
                }
            }
        }
        return TotalLoss;
    }

    // numerical_gradient_shared with this layout (and its point-by-point
    // fallback through loss()).
    __device__ __forceinline__ void gradient(const float *Ininf, float *grad) const {
        enum { NE = 2 * P };
        float v[NE][P];
        const bool share = gradient_points<KIND>(Ininf, v);
        if (!__all_sync(__activemask(), share)) {
            float tI[P];
#pragma unroll
            for (int c = 0; c < P; c++) tI[c] = Ininf[c];
            for (int k = 0; k < P; k++) {
                tI[k] = tI[k] - 0.002f;
                const float tn = loss(tI);
                tI[k] = tI[k] + 0.004f;
                const float tp = loss(tI);
                grad[k] = (tp - tn) * 250.0f;
                tI[k] = tI[k] - 0.002f;
            }
            return;
        }
        float tot[NE];
#pragma unroll
        for (int j = 0; j < NE; j++) tot[j] = 0;
        float rowpos = 0.5f;
#pragma unroll 1
        for (int row = 0; row < R; row++) {
            float w[FULL ? R : M::C4 * 4];
            if constexpr (UNROLL) mask_row(row, w);
#pragma unroll(UNROLL ? R : 1)
            for (int col = 0; col < R; col++) {
                const float2 pl = img[(row * R + col) * ld];
                const float wk = UNROLL ? w[wcol(col)] : mask_at(row, col);
                const float colpos = col + 0.5f;
                const float e_base = single_expo<KIND, DIST>(colpos, rowpos, v[0]);
#pragma unroll
                for (int j = 0; j < NE; j++) {
                    const bool base = (j < 2) || (j >= NE - 2);
                    const float e = base ? e_base : single_expo<KIND, DIST>(colpos, rowpos, v[j]);
                    tot[j] = __fmaf_rn(wk, single_term<KIND>(e, v[j], pl.x, pl.y), tot[j]);
                }
            }
            rowpos += 1.0f;
        }
#pragma unroll
        for (int k = 0; k < P; k++) grad[k] = (tot[2 * k + 1] - tot[2 * k]) * 250.0f;
    }
};

// Pixels of S slots (threads) for PairEval: per row R / 2 column pairs as
// float4 (value, value, log, log), [row][pair][slot], then the last column's
// (value, log) pairs, [row][slot]; 2 R^2 floats per slot in all.
template <int R>
struct PairPixels {
    enum { NP = R / 2, SINGLES = R * NP * 4 };  // SINGLES: floats per slot before the last columns
    __host__ __device__ static constexpr int value(int k, int slot, int S) {
        const int row = k / R, col = k - (k / R) * R;
        return col < 2 * NP ? ((row * NP + col / 2) * S + slot) * 4 + (col & 1) : SINGLES * S + (row * S + slot) * 2;
    }
    // offset of a pixel's log from its value
    __host__ __device__ static constexpr int log_off(int k) { return k - (k / R) * R < 2 * NP ? 2 : 1; }
};

// StagedEval's loss and gradient with the pixels in column pairs (PairPixels)
// and the arithmetic of a pair, or of a parameter's two difference points, in
// packed instructions, exp and log in their flushing forms where flush_safe
// says that this changes nothing.  Term for term the values of StagedEval.
// StagedEval's sums are bound by the issue slots (22.8 instructions a pixel,
// 85% issue, 61% of the special-function pipe); these issue 9.8 and are bound
// by the special-function pipe (79%, two operations of 8 cycles a pixel and
// warp).  100,000 fits in one launch: GS2D 7x7 715 -> 508 us, AS3D 9x9 1645 ->
// 1214 us, GS2D 11x11 1823 -> 1292 us; 600,000 GS2D 7x7 3.72 -> 2.64 ms.  Of
// the line search's evaluations 1.8% (GS2D) run in warps where some ROI is not
// flush_safe (background clamped to zero) and take loss_general.
// pix: this thread's slot of PairPixels, ld the slots.
template <int R, int KIND, int DIST, bool FULL = false>
struct PairEval : MaskView<R, FULL> {
    typedef KindTraits<KIND> T;
    typedef MaskShape<R> M;
    typedef MaskView<R, FULL> V;
    using V::ld;
    using V::mask_row;
    using V::wcol;
    enum { P = T::P, NP = PairPixels<R>::NP, NW = FULL ? R : M::C4 * 4 };
    static_assert(DIST == kFuseFirst || DIST == kFuseSecond, "a fixed distance rounding");
    static_assert(KIND == kGS2D || DIST == kFuseFirst, "AS3D: the x term fused");
    const float4 *pairs;
    const float2 *last;
    __device__ __forceinline__ PairEval(const float *pix, const float *mask_, int slot, int ld_)
        : V{mask_, ld_}, pairs(reinterpret_cast<const float4 *>(pix) + slot),
          last(reinterpret_cast<const float2 *>(pix + PairPixels<R>::SINGLES * ld_) + slot) {}
    __device__ __forceinline__ float2 pixel(int row, int col) const {
        if (col == R - 1) return last[row * ld];
        const float4 q = pairs[(row * NP + col / 2) * ld];
        return (col & 1) ? make_float2(q.y, q.w) : make_float2(q.x, q.z);
    }

    // the packed deviance terms of two pixels or points with models I
    __device__ __forceinline__ static f32x2 terms(f32x2 I, f32x2 pix, f32x2 logpix, f32x2 nln2) {
        // single_term's ln I - ln n is one fused multiply-add, lg2 I * ln 2 - ln n; here its negation
        return fma2(pix, fma2(lg2_flush2(I), nln2, logpix), sub2(I, pix));
    }

    __device__ __forceinline__ float loss(float *v) const {
#pragma unroll
        for (int k = 0; k < P; k++) {
            if (T::CLAMP001) {
                if (v[k] < 0.01f) v[k] = 0.01f;
            } else {
                if (v[k] < 0.0f) v[k] = 0.0f;
            }
        }
        if (!__all_sync(__activemask(), flush_safe<R, KIND>(v))) return loss_general(v);
        const float A = v[0] * QCS_ASCALE, B = v[P - 1] * QCS_BSCALE;
        const f32x2 A2 = pack2(A, A), B2 = pack2(B, B), nln2 = pack2(-kLn2, -kLn2);
        const f32x2 s01 = pack2(QCS_SSCALE, QCS_SSCALE), l2e = pack2(kLog2E, kLog2E), nl2e = pack2(-kLog2E, -kLog2E);
        const f32x2 nS = pack2(-v[3], -v[3]);
        // the column's part of the exponent: dx, dx^2 or dx^2 Sx
        float cx[R];
#pragma unroll
        for (int col = 0; col < R; col++) {
            const float dx = (col + 0.5f) - v[1];
            cx[col] = KIND == kAS3D ? __fmul_rn(__fmul_rn(dx, dx), v[3]) : (DIST == kFuseFirst ? dx : __fmul_rn(dx, dx));
        }
        float total = 0.0f, rowpos = 0.5f;
        const float4 *pr = pairs;
        const float2 *lr = last;
        // rows overlap two at a time (7x7: all): 1-4% over one row at a time
#pragma unroll(R <= 7 ? R : 2)
        for (int row = 0; row < R; row++) {
            float w[NW];
            mask_row(row, w);
            const float dy = rowpos - v[2];
            const float ry = KIND == kAS3D ? __fmul_rn(__fmul_rn(__fmul_rn(dy, dy), v[P - 2]), QCS_SSCALE)
                                           : (DIST == kFuseFirst ? __fmul_rn(dy, dy) : dy);
            const f32x2 ry2 = pack2(ry, ry);
#pragma unroll
            for (int p = 0; p < NP; p++) {
                const float4 q = pr[p * ld];
                const f32x2 c2 = pack2(cx[2 * p], cx[2 * p + 1]), pix = pack2(q.x, q.y), lp = pack2(q.z, q.w);
                f32x2 t;
                if (KIND == kAS3D)
                    t = mul2(fma2(c2, s01, ry2), nl2e);
                else
                    t = mul2(mul2(mul2(DIST == kFuseFirst ? fma2(c2, c2, ry2) : fma2(ry2, ry2, c2), nS), s01), l2e);
                float a, b;
                unpack2(terms(fma2(A2, ex2_flush2(t), B2), pix, lp, nln2), a, b);
                total = __fmaf_rn(w[wcol(2 * p)], a, total);
                total = __fmaf_rn(w[wcol(2 * p + 1)], b, total);
            }
            {
                const float2 q = lr[0];
                float t;
                if (KIND == kAS3D)
                    t = __fmul_rn(__fmaf_rn(cx[R - 1], QCS_SSCALE, ry), -kLog2E);
                else
                    t = __fmul_rn(__fmul_rn(__fmul_rn(DIST == kFuseFirst ? __fmaf_rn(cx[R - 1], cx[R - 1], ry)
                                                                         : __fmaf_rn(ry, ry, cx[R - 1]), -v[3]),
                                            QCS_SSCALE), kLog2E);
                const float I = __fmaf_rn(A, ex2_flush(t), B);
                const float a = __fmaf_rn(lg2_flush(I), -kLn2, q.y);
                total = __fmaf_rn(w[wcol(R - 1)], __fmaf_rn(q.x, a, __fsub_rn(I, q.x)), total);
            }
            rowpos += 1.0f;
            pr += NP * ld;
            lr += ld;
        }
        return total;
    }

    // the same loss with __expf and __logf, at a clamped v
    __device__ __forceinline__ float loss_general(const float *v) const {
        float dxs[R];
#pragma unroll
        for (int col = 0; col < R; col++) dxs[col] = (col + 0.5f) - v[1];
        float total = 0.0f, rowpos = 0.5f;
#pragma unroll 1
        for (int row = 0; row < R; row++) {
            float w[NW];
            mask_row(row, w);
            const float dy = rowpos - v[2];
#pragma unroll
            for (int col = 0; col < R; col++) {
                const float2 pl = pixel(row, col);
                total = __fmaf_rn(w[wcol(col)], single_term<KIND>(single_expo_d<KIND, DIST>(dxs[col], dy, v), v, pl.x, pl.y),
                                  total);
            }
            rowpos += 1.0f;
        }
        return total;
    }

    // The central differences in one sweep over the pixels, the two points of a
    // parameter in one packed value.  The amplitude's points have the same
    // exponential, and so have the background's (the parameters between them
    // are not moved back exactly, so the two differ): 2 (P - 1) exponentials a
    // pixel instead of 2P.
    __device__ __forceinline__ void gradient(const float *Ininf, float *grad) const {
        enum { NE = 2 * P };
        float v[NE][P];
        gradient_points<KIND>(Ininf, v);
        bool ok = true;
#pragma unroll
        for (int j = 0; j < NE; j++)
            ok = ok && v[j][P - 1] * QCS_BSCALE >= fmaxf(1e-30f, v[j][0] * QCS_ASCALE * 0x1p-90f);  // flush_safe
        if (!__all_sync(__activemask(), ok)) {
            float tot[NE];
#pragma unroll 1
            for (int j = 0; j < NE; j++) {
                float x[P];
#pragma unroll
                for (int c = 0; c < P; c++) {
                    x[c] = v[0][c];
#pragma unroll
                    for (int i = 1; i < NE; i++) x[c] = j == i ? v[i][c] : x[c];
                }
                const float f = loss_general(x);
#pragma unroll
                for (int i = 0; i < NE; i++) tot[i] = j == i ? f : (j == 0 ? 0.0f : tot[i]);
            }
#pragma unroll
            for (int k = 0; k < P; k++) grad[k] = (tot[2 * k + 1] - tot[2 * k]) * 250.0f;
            return;
        }
        const f32x2 nln2 = pack2(-kLn2, -kLn2), s01 = pack2(QCS_SSCALE, QCS_SSCALE);
        const f32x2 l2e = pack2(kLog2E, kLog2E), nl2e = pack2(-kLog2E, -kLog2E);
        f32x2 tot[P], A2[P], B2[P];
#pragma unroll
        for (int k = 0; k < P; k++) {
            tot[k] = pack2(0.0f, 0.0f);
            A2[k] = pack2(v[2 * k][0] * QCS_ASCALE, v[2 * k + 1][0] * QCS_ASCALE);
            B2[k] = pack2(v[2 * k][P - 1] * QCS_BSCALE, v[2 * k + 1][P - 1] * QCS_BSCALE);
        }
        // exponential pair q: the amplitude's and the background's (q = 0), else parameter q's two points
        auto lo = [&](int q, int c) { return v[q == 0 ? 0 : 2 * q][c]; };
        auto hi = [&](int q, int c) { return v[q == 0 ? NE - 1 : 2 * q + 1][c]; };
        float rowpos = 0.5f;
#pragma unroll 1
        for (int row = 0; row < R; row++) {
            float w[NW];
            mask_row(row, w);
            // the row's part of each exponent
            auto row_part = [&](float y, float Sy) {
                const float dy = rowpos - y;
                return KIND == kAS3D ? __fmul_rn(__fmul_rn(__fmul_rn(dy, dy), Sy), QCS_SSCALE)
                                     : (DIST == kFuseFirst ? __fmul_rn(dy, dy) : dy);
            };
            f32x2 ry[P - 1];
#pragma unroll
            for (int q = 0; q < P - 1; q++)
                ry[q] = pack2(row_part(lo(q, 2), lo(q, P - 2)), row_part(hi(q, 2), hi(q, P - 2)));
#pragma unroll
            for (int col = 0; col < R; col++) {
                const float2 pl = pixel(row, col);
                const float wk = w[wcol(col)];
                const f32x2 pix = pack2(pl.x, pl.x), lp = pack2(pl.y, pl.y), w2 = pack2(wk, wk);
                f32x2 e[P - 1];
#pragma unroll
                for (int q = 0; q < P - 1; q++) {
                    const f32x2 dx = pack2((col + 0.5f) - lo(q, 1), (col + 0.5f) - hi(q, 1));
                    f32x2 t;
                    if (KIND == kAS3D) {
                        const f32x2 Sx = pack2(lo(q, 3), hi(q, 3));
                        t = mul2(fma2(mul2(mul2(dx, dx), Sx), s01, ry[q]), nl2e);
                    } else {
                        const f32x2 nS = pack2(-lo(q, 3), -hi(q, 3));
                        t = mul2(mul2(mul2(DIST == kFuseFirst ? fma2(dx, dx, ry[q]) : fma2(ry[q], ry[q], mul2(dx, dx)), nS),
                                      s01), l2e);
                    }
                    e[q] = ex2_flush2(t);
                }
                float e_first, e_last;
                unpack2(e[0], e_first, e_last);
#pragma unroll
                for (int k = 0; k < P; k++) {
                    const f32x2 ek = k == 0 ? pack2(e_first, e_first) : (k == P - 1 ? pack2(e_last, e_last) : e[k]);
                    tot[k] = fma2(w2, terms(fma2(A2[k], ek, B2[k]), pix, lp, nln2), tot[k]);
                }
            }
            rowpos += 1.0f;
        }
#pragma unroll
        for (int k = 0; k < P; k++) {
            float n, p;
            unpack2(tot[k], n, p);
            grad[k] = (p - n) * 250.0f;
        }
    }
};

// The single-emitter evaluator of a thread: packed where the distance's
// rounding is fixed in the source.
template <int R, int DIST>
constexpr bool kPaired = DIST != kCompiler && R <= kUnrollMaxR;

// The learned-start single fit's loss and analytic gradient over the staged
// layout of fit_single_kernel (pixels as (value, log) pairs, the mask's unique
// values): StagedEval's loss, the gradient of AnalyticEvalGS2D /
// AnalyticEvalAS3D term for term (the mask values are the same, so the
// results are those of the full-mask evaluators).
template <int R, int KIND, class B, bool FULL>
struct StagedAnalyticEval : B {
    using B::B;
    __device__ __forceinline__ void gradient(const float *v, float *g) const {
        enum { NW = FULL ? R : B::M::C4 * 4 };
        if constexpr (KIND == kGS2D) {
            float c[5];
#pragma unroll
            for (int k = 0; k < 5; k++) c[k] = v[k] < 0.0f ? 0.0f : v[k];
            const float A128 = c[0] * QCS_ASCALE, B64 = c[4] * QCS_BSCALE, S01 = c[3] * QCS_SSCALE;
            float gA = 0, gX = 0, gY = 0, gS = 0, gB = 0;
#pragma unroll 1
            for (int row = 0; row < R; row++) {
                float wr[NW];
                this->mask_row(row, wr);
                const float dy = (row + 0.5f) - c[2];
#pragma unroll(R <= kUnrollMaxR ? R : 1)
                for (int col = 0; col < R; col++) {
                    const float2 pl = this->pixel(row, col);
                    const float w = wr[B::wcol(col)];
                    const float dx = (col + 0.5f) - c[1];
                    const float r2 = __fmaf_rn(dx, dx, dy * dy);
                    const float e = __expf(-r2 * S01);
                    const float mu = __fmaf_rn(A128, e, B64);
                    const float q = w * (1.0f - __fdividef(pl.x, mu));
                    const float qe = q * e;
                    gA += qe;
                    gX = __fmaf_rn(qe, dx, gX);
                    gY = __fmaf_rn(qe, dy, gY);
                    gS = __fmaf_rn(qe, r2, gS);
                    gB += q;
                }
            }
            g[0] = QCS_ASCALE * gA;
            g[1] = A128 * 2.0f * S01 * gX;
            g[2] = A128 * 2.0f * S01 * gY;
            g[3] = -A128 * QCS_SSCALE * gS;
            g[4] = QCS_BSCALE * gB;
        } else {
            float c[6];
#pragma unroll
            for (int k = 0; k < 6; k++) c[k] = v[k] < 0.01f ? 0.01f : v[k];
            const float A128 = c[0] * QCS_ASCALE, B64 = c[5] * QCS_BSCALE;
            const float Sx = c[3] * QCS_SSCALE, Sy = c[4] * QCS_SSCALE;
            float gA = 0, gX = 0, gY = 0, gSx = 0, gSy = 0, gB = 0;
#pragma unroll 1
            for (int row = 0; row < R; row++) {
                float wr[NW];
                this->mask_row(row, wr);
                const float dy = (row + 0.5f) - c[2];
                const float qy = dy * dy;
#pragma unroll(R <= kUnrollMaxR ? R : 1)
                for (int col = 0; col < R; col++) {
                    const float2 pl = this->pixel(row, col);
                    const float w = wr[B::wcol(col)];
                    const float dx = (col + 0.5f) - c[1];
                    const float qx = dx * dx;
                    const float e = __expf(-__fmaf_rn(qx, Sx, qy * Sy));
                    const float mu = __fmaf_rn(A128, e, B64);
                    const float q = w * (1.0f - __fdividef(pl.x, mu));
                    const float qe = q * e;
                    gA += qe;
                    gX = __fmaf_rn(qe, dx, gX);
                    gY = __fmaf_rn(qe, dy, gY);
                    gSx = __fmaf_rn(qe, qx, gSx);
                    gSy = __fmaf_rn(qe, qy, gSy);
                    gB += q;
                }
            }
            g[0] = QCS_ASCALE * gA;
            g[1] = A128 * 2.0f * Sx * gX;
            g[2] = A128 * 2.0f * Sy * gY;
            g[3] = -A128 * QCS_SSCALE * gSx;
            g[4] = -A128 * QCS_SSCALE * gSy;
            g[5] = QCS_BSCALE * gB;
        }
    }
};

// Fixed schedule: IT quasi-Newton iterations, each with an NB-step bisection
// of the step length in [1e-5, 1] (the reference: 11); no convergence test.
// D: P x P scratch at D[(r * P + c) * ld]; ev evaluates the loss and the
// gradient.
template <int P, int IT, class Eval, int NB = kBisections>
__device__ __forceinline__ void bfgs_fit(const Eval &ev, float *Ininf, float *D, int ld) {
    float grad[P], d0[P], td0[P], sk[P], yk[P], tgrad[P];
    float ddat[2], dpos[2];  // two-element arrays indexed by constants only
#pragma unroll
    for (int r = 0; r < P; r++) {
#pragma unroll
        for (int c = 0; c < P; c++) D[(r * P + c) * ld] = (r == c) ? 1.0f : 0.0f;
    }
    ev.gradient(Ininf, grad);
#pragma unroll
    for (int rcnt = 0; rcnt < P; rcnt++) d0[rcnt] = -grad[rcnt];

    for (int itcnt = 0; itcnt < IT; itcnt++) {
        float td0_total = 0;
#pragma unroll
        for (int rcnt = 0; rcnt < P; rcnt++) {
            td0[rcnt] = fabsf(d0[rcnt]);
            td0_total += td0[rcnt];
        }
        td0_total = ((float)P) / td0_total;
#pragma unroll
        for (int rcnt = 0; rcnt < P; rcnt++) d0[rcnt] = d0[rcnt] * td0_total;

        dpos[0] = 0.00001f;
        dpos[1] = 1.0f;
        {
            float xlo[P], xhi[P];
#pragma unroll
            for (int cnt = 0; cnt < P; cnt++) xlo[cnt] = d0[cnt] * 0.0001f + Ininf[cnt];
#pragma unroll
            for (int cnt = 0; cnt < P; cnt++) xhi[cnt] = d0[cnt] * 1.0f + Ininf[cnt];
            ddat[0] = ev.loss(xlo);
            ddat[1] = ev.loss(xhi);
        }

        // Bisection: the half that moves is chosen per ROI; the moved point
        // is built with a select so that every thread of a warp runs the same
        // single loss evaluation (no divergent branches around the loss).
        for (int cnt = 0; cnt < NB; cnt++) {
            const int xdsel = (ddat[0] < ddat[1]);
            const float mid = (dpos[0] + dpos[1]) * 0.5f;
            dpos[0] = xdsel ? dpos[0] : mid;
            dpos[1] = xdsel ? mid : dpos[1];
            if (cnt < NB - 1) {
                const float dsel = xdsel ? dpos[1] : dpos[0];
                float xn[P];
#pragma unroll
                for (int k = 0; k < P; k++) xn[k] = d0[k] * dsel + Ininf[k];
                const float f = ev.loss(xn);
                ddat[0] = xdsel ? ddat[0] : f;
                ddat[1] = xdsel ? f : ddat[1];
            }
        }
        const float scale = (dpos[0] + dpos[1]) * 0.5f;
#pragma unroll
        for (int rcnt = 0; rcnt < P; rcnt++) {
            sk[rcnt] = d0[rcnt] * scale;
            Ininf[rcnt] = Ininf[rcnt] + sk[rcnt];
        }
#pragma unroll
        for (int cnt = 0; cnt < P; cnt++)
            if (Ininf[cnt] < 0.01f) Ininf[cnt] = 0.01f;

        if (itcnt < IT - 1) {
#pragma unroll
            for (int rcnt = 0; rcnt < P; rcnt++) tgrad[rcnt] = grad[rcnt];
            ev.gradient(Ininf, grad);
#pragma unroll
            for (int rcnt = 0; rcnt < P; rcnt++) yk[rcnt] = grad[rcnt] - tgrad[rcnt];
            bfgs_update<P>(D, ld, sk, yk);
#pragma unroll
            for (int row = 0; row < P; row++) {
                d0[row] = 0;
#pragma unroll
                for (int cnt = 0; cnt < P; cnt++) d0[row] -= D[(row * P + cnt) * ld] * grad[cnt];
            }
        }
    }
}

// bfgs_update with few live registers, for one lane that updates an inverse
// Hessian shared by a lane group: D (row-major P x P) and the scratch T
// (P x P) in shared memory.  The same values as bfgs_update, operation for
// operation: its P x P temporaries are recomputed from sk and the scaled
// vectors with the roundings nvcc gives their expressions (one fused
// multiply-add or separate product each), the left product kept in T.
// SKSK_FUSED: the final D + sk sk'/(y's) fused into one multiply-add (nvcc
// may contract the separately computed product into the sum).
template <int P, bool SKSK_FUSED>
__device__ __forceinline__ void bfgs_update_light(float *D, float *T, const float *sk, const float *yk) {
    float divdat = 0;
#pragma unroll
    for (int cnt = 0; cnt < P; cnt++) divdat = __fmaf_rn(sk[cnt], yk[cnt], divdat);
    divdat = 1.0f / divdat;
    float tdat10[P], tdat20[P];
#pragma unroll
    for (int cnt = 0; cnt < P; cnt++) {
        tdat10[cnt] = __fmul_rn(yk[cnt], divdat);
        tdat20[cnt] = __fmul_rn(sk[cnt], divdat);
    }
    // skyk(r, c) = [r == c] - sk[r] tdat10[c], one rounding
    auto skyk = [&](int r, int c) { return __fmaf_rn(-sk[r], tdat10[c], r == c ? 1.0f : 0.0f); };
#pragma unroll 1
    for (int row = 0; row < P; row++) {
#pragma unroll
        for (int col = 0; col < P; col++) {
            float acc = 0;
#pragma unroll
            for (int cnt = 0; cnt < P; cnt++) acc = __fmaf_rn(skyk(row, cnt), D[cnt * P + col], acc);
            T[row * P + col] = acc;
        }
    }
#pragma unroll 1
    for (int row = 0; row < P; row++) {
#pragma unroll
        for (int col = 0; col < P; col++) {
            float acc = 0;
#pragma unroll
            for (int cnt = 0; cnt < P; cnt++) acc = __fmaf_rn(T[row * P + cnt], skyk(col, cnt), acc);
            D[row * P + col] = SKSK_FUSED ? __fmaf_rn(sk[row], tdat20[col], acc)
                                          : __fadd_rn(acc, __fmul_rn(sk[row], tdat20[col]));
        }
    }
}

// bfgs_fit for a lane group that shares one inverse Hessian per ROI: every
// lane runs the line search and the evaluations (which need all lanes), the
// group's first lane alone updates D (bfgs_update_light) and the new search
// direction, which the others then read from dbuf.  D, T: P x P, dbuf: P
// floats of shared memory per ROI.  The same values as bfgs_fit.
template <int P, int IT, class Eval, bool SKSK_FUSED, int NB = kBisections>
__device__ __forceinline__ void bfgs_fit_shared(const Eval &ev, float *Ininf, float *D, float *T, float *dbuf,
                                                int lane, unsigned mask) {
    float grad[P], d0[P], td0[P], sk[P], yk[P], tgrad[P];
    float ddat[2], dpos[2];
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < P; r++) {
#pragma unroll
            for (int c = 0; c < P; c++) D[r * P + c] = (r == c) ? 1.0f : 0.0f;
        }
    }
    ev.gradient(Ininf, grad);
#pragma unroll
    for (int rcnt = 0; rcnt < P; rcnt++) d0[rcnt] = -grad[rcnt];

    for (int itcnt = 0; itcnt < IT; itcnt++) {
        float td0_total = 0;
#pragma unroll
        for (int rcnt = 0; rcnt < P; rcnt++) {
            td0[rcnt] = fabsf(d0[rcnt]);
            td0_total += td0[rcnt];
        }
        td0_total = ((float)P) / td0_total;
#pragma unroll
        for (int rcnt = 0; rcnt < P; rcnt++) d0[rcnt] = d0[rcnt] * td0_total;

        dpos[0] = 0.00001f;
        dpos[1] = 1.0f;
        {
            float xlo[P], xhi[P];
#pragma unroll
            for (int cnt = 0; cnt < P; cnt++) xlo[cnt] = d0[cnt] * 0.0001f + Ininf[cnt];
#pragma unroll
            for (int cnt = 0; cnt < P; cnt++) xhi[cnt] = d0[cnt] * 1.0f + Ininf[cnt];
            ddat[0] = ev.loss(xlo);
            ddat[1] = ev.loss(xhi);
        }
        for (int cnt = 0; cnt < NB; cnt++) {
            const int xdsel = (ddat[0] < ddat[1]);
            const float mid = (dpos[0] + dpos[1]) * 0.5f;
            dpos[0] = xdsel ? dpos[0] : mid;
            dpos[1] = xdsel ? mid : dpos[1];
            if (cnt < NB - 1) {
                const float dsel = xdsel ? dpos[1] : dpos[0];
                float xn[P];
#pragma unroll
                for (int k = 0; k < P; k++) xn[k] = d0[k] * dsel + Ininf[k];
                const float f = ev.loss(xn);
                ddat[0] = xdsel ? ddat[0] : f;
                ddat[1] = xdsel ? f : ddat[1];
            }
        }
        const float scale = (dpos[0] + dpos[1]) * 0.5f;
#pragma unroll
        for (int rcnt = 0; rcnt < P; rcnt++) {
            sk[rcnt] = d0[rcnt] * scale;
            Ininf[rcnt] = Ininf[rcnt] + sk[rcnt];
        }
#pragma unroll
        for (int cnt = 0; cnt < P; cnt++)
            if (Ininf[cnt] < 0.01f) Ininf[cnt] = 0.01f;

        if (itcnt < IT - 1) {
#pragma unroll
            for (int rcnt = 0; rcnt < P; rcnt++) tgrad[rcnt] = grad[rcnt];
            ev.gradient(Ininf, grad);
            if (lane == 0) {
#pragma unroll
                for (int rcnt = 0; rcnt < P; rcnt++) yk[rcnt] = grad[rcnt] - tgrad[rcnt];
                bfgs_update_light<P, SKSK_FUSED>(D, T, sk, yk);
#pragma unroll
                for (int row = 0; row < P; row++) {
                    float acc = 0;
#pragma unroll
                    for (int cnt = 0; cnt < P; cnt++) acc = __fmaf_rn(-D[row * P + cnt], grad[cnt], acc);
                    dbuf[row] = acc;
                }
            }
            __syncwarp(mask);
#pragma unroll
            for (int row = 0; row < P; row++) d0[row] = dbuf[row];
            __syncwarp(mask);
        }
    }
}

template <int R, int KIND, int DIST = ArithSpec<KIND, R>::DIST, int SUM2 = ArithSpec<KIND, R>::SUM2,
          int ITERS = KindTraits<KIND>::IT>
__device__ __forceinline__ void mle_fit(const RoiRef &roi, float *Ininf, float *D, int ld) {
    bfgs_fit<KindTraits<KIND>::P, ITERS>(ThreadEval<R, KIND, DIST, SUM2>{roi}, Ininf, D, ld);
}

// One pixel's weight of the mask below, for the sizes whose contraction is fixed in the source.
template <int R, int MASK>
__device__ __forceinline__ float wle_weight(float colpos, float rowpos, float WLE_SigmaX, float WLE_SigmaY,
                                            int MoleculeType) {
    const float ROICenter = R / 2.0f;
    const float WLE_SigmaX1 = 1.0f / (2.0f * WLE_SigmaX * WLE_SigmaX);
    const float WLE_SigmaY1 = 1.0f / (2.0f * WLE_SigmaY * WLE_SigmaY);
    if (MoleculeType == 0) return 1.0f;
    return __expf(-sum_of_products<MASK>((colpos - ROICenter) * (colpos - ROICenter), WLE_SigmaX1,
                                         (rowpos - ROICenter) * (rowpos - ROICenter), WLE_SigmaY1));
}

// Weighted-MLE mask (bfgsMLE_core.h:206-238).
template <int R, int MASK = kCompiler>
__device__ __forceinline__ void wle_weights(float *w, int ld, float WLE_SigmaX, float WLE_SigmaY, int MoleculeType) {
    const float ROICenter = R / 2.0f;
    const float WLE_SigmaX1 = 1.0f / (2.0f * WLE_SigmaX * WLE_SigmaX);
    const float WLE_SigmaY1 = 1.0f / (2.0f * WLE_SigmaY * WLE_SigmaY);
    for (int row = 0; row < R; row++) {
        for (int col = 0; col < R; col++) {
            const float rowpos = row + 0.5f;
            const float colpos = col + 0.5f;
            if (MoleculeType == 0)
                w[(row * R + col) * ld] = 1.0f;
            else
                w[(row * R + col) * ld] =
                    __expf(-sum_of_products<MASK>((colpos - ROICenter) * (colpos - ROICenter), WLE_SigmaX1,
                                                  (rowpos - ROICenter) * (rowpos - ROICenter), WLE_SigmaY1));
        }
    }
}

}  // namespace qcs
