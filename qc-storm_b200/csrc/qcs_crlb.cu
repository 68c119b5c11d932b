// CRLB of x and y for each localization: diagonal Fisher information from
// numerical second derivatives (dh = 0.02) of a Gaussian PSF model on a fixed
// 9x9 (2D) or 15x15 (astigmatic 3D) grid with the emitter at the centre, the
// fitted total photons, background (+ read noise^2) and sigma x/y;
// CRLB = PixelSize / sqrt(FI) in nm, 100 when the row is not fittable.
// Re-expressed from LocPrecCalc_GaussianCRLB.h:65-243 with every rounding
// step explicit (bit-identical results at 9 x 9); adds the bounds guard that
// the reference kernel lacks (:65-128) and reads the row count from the
// device.
#include <cuda_runtime.h>

#include "qcs_fit_math.cuh"
#include "qcs_kernels.h"

namespace qcs {
namespace {

// Contraction of the PSF exponent dx^2/(2 sx^2) + dy^2/(2 sy^2) at each of
// the reference's evaluation sites, as nvcc compiles GaussianPSF_generate2D
// inlined into them (found by comparing every combination against the
// reference's CUDA build; see SumMode in qcs_fit_math.cuh): CENTRE = the
// model and the base point of both derivatives (x0 = y0 = 0), SHIFT_X = the
// +-dh points of the x derivative, SHIFT_Y = those of the y derivative.
// PeakPn * exp(.) + background and d2 - model * d2log are fused
// multiply-adds at every site.
template <int G>
struct CrlbSites;
template <>
struct CrlbSites<9> {
    enum { CENTRE = kFuseSecond, SHIFT_X = kFuseFirst, SHIFT_Y = kFuseSecond };
};
template <>
struct CrlbSites<15> {
    enum { CENTRE = kFuseFirst, SHIFT_X = kFuseFirst, SHIFT_Y = kFuseSecond };
};

struct PsfPara {
    float peak, six, siy, bkg;
};

// Gaussian PSF value of the reference's model at offsets dx = CurX - x0,
// dy = CurY - y0 (LocPrecCalc_GaussianCRLB.h:131-173).
template <int MODE>
__device__ __forceinline__ float psf_value(const PsfPara &p, float dx, float dy) {
    const float e = __expf(-sum_of_products<MODE>(__fmul_rn(dx, dx), p.six, __fmul_rn(dy, dy), p.siy));
    return __fmaf_rn(p.peak, e, p.bkg);
}

// x / 0.02f correctly rounded without a division: with C the double-length
// reciprocal ch + cl of 0.02f, RN(ch x + RN(cl x)) (Brisebarre and Muller,
// "Correctly rounded multiplication by arbitrary precision constants", IEEE
// Trans. Comput. 57, 2008).  Compared with the division for every float in the
// range it is used for (a zero may lose its sign, which no sum shows).
__device__ __forceinline__ float div_dh(float x) {
    constexpr double inv = 1.0 / (double)0.02f;
    constexpr float ch = (float)inv, cl = (float)(inv - (double)ch);
    const float q = __fmaf_rn(ch, x, __fmul_rn(cl, x));
    const float a = fabsf(x);
    if (a < 1e30f && (a > 1e-30f || a == 0.0f)) return q;
    return __fdiv_rn(x, 0.02f);
}

// (f(+h) - 2 f(0) + f(-h)) / h / h with the reference's rounding
// (LocPrecCalc_GaussianCRLB.h:188-196; 2 f(0) is exact, so fusing it changes nothing).
__device__ __forceinline__ float second_diff(float fp, float f0, float fn) {
    return div_dh(div_dh(__fadd_rn(__fmaf_rn(-2.0f, f0, fp), fn)));
}

// Rows per block.
__host__ __device__ constexpr int crlb_rows(int G) { return G == 9 ? 32 : 16; }

// One thread per row, axis and line of the half grid.  The reference
// evaluates the PSF on the full grid seven times per row (model, then base,
// +dh, -dh for each derivative) and sums d2 - model * d2log over every pixel.
// The same values come from far fewer evaluations, exactly: the base points
// equal the model (same parameters, same rounding), the model is symmetric in
// x and y, the -dh evaluation is the +dh one mirrored (x - (-h) = -((-x) - h)
// exactly), and each derivative's terms are symmetric across the other axis.
// So a thread takes one line: its model values (half a line) and +dh values,
// then its terms, kept in shared memory ([term][row and axis]); after a
// barrier one thread per row and axis adds every pixel's term in the
// reference's pixel order.  The y terms are the x terms with the axes
// exchanged (the reference's two sites contract mirror-image products); a
// warp holds one axis of 32 rows (15 x 15: two axes of 16).  100,000 rows at 9
// x 9: 41 us, 60,013 at 15 x 15: 67, 300 at 9 x 9: 6 (a thread per row and
// axis walking the lines: 43, 92, 13; two lanes per row sharing a model table,
// with divisions: 66, 221, 24).  Bound by the instructions of logf, Q +
// G a line.
template <int G>
__global__ void __launch_bounds__((G / 2 + 1) * (G == 9 ? 64 : 32)) crlb_kernel(
    float *__restrict__ loc, const int *__restrict__ n_dev, int n, const int *__restrict__ ids,
    const uint8_t *__restrict__ skip, float ReadNoise_e, float QE, float PixelSize) {
    enum { H = G / 2, Q = H + 1, ROWS = crlb_rows(G), LANES = 2 * ROWS };
    using S = CrlbSites<G>;
    // the x-derivative thread uses fma(dx^2, six, dy^2 siy), the y-derivative thread
    // fma(dy^2, siy, dx^2 six): one expression with its operands exchanged
    static_assert(S::SHIFT_X == kFuseFirst && S::SHIFT_Y == kFuseSecond, "mirrored derivative sites");
    __shared__ float sT[Q * G][LANES];
    const int slot = threadIdx.x % LANES, l = threadIdx.x / LANES;
    const int role = slot / ROWS;  // 0: x, 1: y
    const int rows = n_dev ? *n_dev : n;
    const int k_slot = blockIdx.x * ROWS + slot % ROWS;
    if (blockIdx.x * ROWS >= rows) return;  // the whole block
    const int gid = k_slot < rows ? (ids ? ids[k_slot] : k_slot) : 0;
    const bool have = k_slot < rows && !(skip && skip[gid]);
    float *r = loc + (size_t)gid * 12;
    float *T = &sT[0][slot];
    bool valid = false;
    if (have) {
        const float TotalPhoton_e = __fmul_rn(r[QCS_POS_TPHO], QE);
        float Background_e = __fmul_rn(r[QCS_POS_BAKG], QE);
        const float sx = r[QCS_POS_SIGX], sy = r[QCS_POS_SIGY];
        valid = (TotalPhoton_e > 1) && (Background_e > 1) && (sx > 0.1) && (sy > 0.1) && (sx < 10) && (sy < 10);
        if (valid) {
            // read noise counted into the background (LocPrecCalc_GaussianCRLB.h:89-92)
            Background_e = __fdiv_rn(__fmaf_rn(ReadNoise_e, ReadNoise_e, __fmul_rn(Background_e, QE)), QE);
            const float pi = 3.141592654f;
            PsfPara p;
            p.peak = __fmul_rn(__fdiv_rn(1.0f, __fmul_rn(__fmul_rn(__fmul_rn(2.0f, pi), sx), sy)), TotalPhoton_e);
            p.six = __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, sx), sx));
            p.siy = __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, sy), sy));
            p.bkg = Background_e;
            const float h = 0.02f;
            const float su = role ? p.siy : p.six, sv = role ? p.six : p.siy;
            // x thread: the +dh row at |CurY| = l, every column k; y thread: the
            // +dh column at |CurX| = l, every row k
            const float fl = (float)l;
            const float ll = __fmul_rn(__fmul_rn(fl, fl), sv);
            float m[Q], lm[Q], tp[G], lp[G];
#pragma unroll
            for (int o = 0; o < Q; ++o) {
                const float dx = role ? fl : (float)o, dy = role ? (float)o : fl;
                m[o] = psf_value<S::CENTRE>(p, dx, dy);
                lm[o] = logf(m[o]);
            }
#pragma unroll
            for (int k = 0; k < G; ++k) {
                const float sh = __fsub_rn((float)(k - H), h);
                tp[k] = __fmaf_rn(p.peak, __expf(-__fmaf_rn(__fmul_rn(sh, sh), su, ll)), p.bkg);
                lp[k] = logf(tp[k]);
            }
#pragma unroll
            for (int k = 0; k < G; ++k) {
                const int o = k < H ? H - k : k - H;  // |k - H|
                const float d2 = second_diff(tp[k], m[o], tp[G - 1 - k]);
                const float dl = second_diff(lp[k], lm[o], lp[G - 1 - k]);
                T[(l * G + k) * LANES] = __fmaf_rn(-m[o], dl, d2);
            }
        }
    }
    __syncthreads();  // the lines' terms; the row is read by all before its CRLB is written
    if (l != 0 || !have) return;
    float std_dev = 100.0f;
    if (valid) {
        // Fisher information, pixel order (LocPrecCalc_GaussianCRLB.h:226-243)
        float F = 0;
#pragma unroll 1
        for (int y = 0; y < G; ++y) {
            const int ay = y < H ? H - y : y - H;
#pragma unroll
            for (int x = 0; x < G; ++x) {
                const int bx = x < H ? H - x : x - H;
                F = __fadd_rn(F, T[(role ? bx * G + y : ay * G + x) * LANES]);
            }
        }
        if (F == 0.0f) F = 1;
        std_dev = __fmul_rn(__fsqrt_rn(__fdiv_rn(1.0f, F)), PixelSize);
    }
    r[role ? QCS_POS_CRBY : QCS_POS_CRBX] = std_dev;
}

}  // namespace

cudaError_t launch_crlb(float *loc, const int *n_dev, int n, int max_rows, int loc_type, float ReadNoise_e, float QE,
                        float PixelSize, cudaStream_t s, const int *ids, const uint8_t *skip) {
    if (max_rows <= 0) return cudaSuccess;
    const int rows = loc_type != QCS_LOCTYPE_AS3D ? crlb_rows(9) : crlb_rows(15);
    const int blocks = (max_rows + rows - 1) / rows;
    if (loc_type != QCS_LOCTYPE_AS3D)
        crlb_kernel<9><<<blocks, 2 * rows * 5, 0, s>>>(loc, n_dev, n, ids, skip, ReadNoise_e, QE, PixelSize);
    else
        crlb_kernel<15><<<blocks, 2 * rows * 8, 0, s>>>(loc, n_dev, n, ids, skip, ReadNoise_e, QE, PixelSize);
    return cudaGetLastError();
}

}  // namespace qcs
