// Evaluators of the fit kernels (qcs_fit_math.cuh) against the general loss
// and gradient, loss() and numerical_gradient(), which call __expf and __logf
// for every pixel.  Built and driven by test_gpu_evaluators.py.
#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>

#include "qcs_fit_math.cuh"

using namespace qcs;

namespace {

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__device__ bool subnormal(float v) { return v != 0.0f && fabsf(v) < 1.17549435e-38f; }

// Over every float x: [0] the flushing exp differs from __expf where that is not
// subnormal, [1] is not zero where it is; [2] the keeping exp differs anywhere;
// [3] the flushing log differs from __logf where x is not subnormal.
__global__ void exp_log_kernel(unsigned long long *out) {
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    unsigned long long bad[4] = {0, 0, 0, 0};
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += step) {
        const float x = __uint_as_float((unsigned)i);
        const float e = __expf(x), t = __fmul_rn(x, kLog2E);
        if (subnormal(e))
            bad[1] += ex2_flush(t) != 0.0f;
        else
            bad[0] += !same(ex2_flush(t), e);
        bad[2] += !same(ex2_keep(t), e);
        if (!subnormal(x)) bad[3] += !same(__fmul_rn(lg2_flush(x), kLn2), __logf(x));
    }
    for (int k = 0; k < 4; ++k)
        if (bad[k]) atomicAdd(out + k, bad[k]);
}

template <int R, int KIND>
constexpr bool kFullMask = (int)ArithSpec<KIND, R>::MASK == (int)kCompiler;

// One ROI of the general side: pixels (value, log) and the mask.
template <int R, int KIND>
__device__ void general_roi(const float *pix, float sigma, float2 *img, float *w) {
    for (int k = 0; k < R * R; ++k) img[k] = make_float2(pix[k], __logf(pix[k]));
    wle_weights<R, ArithSpec<KIND, R>::MASK>(w, 1, sigma, sigma, 1);
}

// Case i by G lanes (LaneFit) and by one thread: the losses at x + d step[j] of
// four steps, then the gradient at x; path[i]: bit j says that loss j may take
// the flushing form.
template <int R, int KIND, int G>
__global__ void __launch_bounds__(32) lanes_kernel(int n, const float *pix, const float *sigma, const float *x,
                                                   const float *d, float2 *img, float *w, float *fast, float *general,
                                                   int *path) {
    typedef LaneLayout<R, KIND> L;
    typedef LaneFit<R, KIND, ArithSpec<KIND, R>::DIST, G> Fit;
    enum { P = KindTraits<KIND>::P, PIX = R * R, OUT = 4 + P };
    extern __shared__ __align__(16) float smem[];
    for (int k = threadIdx.x; k < L::PIXP; k += 32) {
        smem[k] = k % R + 0.5f;
        smem[L::PIXP + k] = k / R + 0.5f;
    }
    const int group = threadIdx.x / G, lane = threadIdx.x % G, i = blockIdx.x * (32 / G) + group;
    if (i >= n) return;  // the last block is whole: n is a multiple of 32 / G
    const unsigned mask = G == 32 ? 0xffffffffu : ((1u << (G % 32)) - 1u) << (threadIdx.x & ~(G - 1));
    float *s = smem + 2 * L::PIXP + group * L::TOTAL;
    img += (size_t)i * PIX;
    w += (size_t)i * PIX;
    if (lane == 0) general_roi<R, KIND>(pix + (size_t)i * PIX, sigma[i], img, w);
    __syncwarp();
    for (int k = lane; k < L::PIXP; k += G) {
        const float v = k < PIX ? pix[(size_t)i * PIX + k] : 1.0f;
        s[L::VAL + k] = v;
        s[L::LOG + k] = __logf(v);
        if (KindTraits<KIND>::WEIGHTED && k < PIX) s[L::W + k] = w[k];
    }
    __syncwarp();
    float xs[P], ds[P], end[P], grad[P], f[4];
    for (int k = 0; k < P; ++k) {
        xs[k] = x[(size_t)i * P + k];
        ds[k] = d[(size_t)i * P + k];
    }
    const float step[4] = {0.0f, 1.0f, 0.0001f, 0.31640625f};
    const Fit fit{smem, s, lane, mask};
    for (int k = 0; k < P; ++k) end[k] = xs[k] + ds[k];
    const bool normal = Fit::exps_normal(xs, end);
    fit.losses(xs, ds, step, normal, f);
    fit.gradient(xs, grad, normal);
    if (lane != 0) return;
    float *o = fast + (size_t)i * OUT, *g = general + (size_t)i * OUT;
    for (int j = 0; j < 4; ++j) o[j] = f[j];
    for (int k = 0; k < P; ++k) o[4 + k] = grad[k];
    const RoiRef roi{img, w, 1};
    int taken = 0;
    for (int j = 0; j < 4; ++j) {
        float v[P];
        for (int k = 0; k < P; ++k) v[k] = __fmaf_rn(ds[k], step[j], xs[k]);
        g[j] = loss<R, KIND>(roi, v);
        taken |= (Fit::safe(v[P - 1], v[0]) && (normal || Fit::exps_normal(v, v))) << j;
    }
    numerical_gradient<R, KIND>(roi, xs, g + 4);
    path[i] = taken;
}

// Case i by its thread (PairEval): the loss at x, then the gradient; path: the
// block's warp took the loss in the flushing form.
template <int R, int KIND>
__global__ void __launch_bounds__(32) pairs_kernel(int n, const float *pix, const float *sigma, const float *x,
                                                   float2 *img, float *w, float *fast, float *general, int *path) {
    typedef ArithSpec<KIND, R> A;
    constexpr bool FULL = kFullMask<R, KIND>;
    static_assert(kPaired<R, A::DIST>, "a size that PairEval evaluates");
    enum { P = KindTraits<KIND>::P, PIX = R * R, OUT = 1 + P, S = 32 };
    extern __shared__ __align__(16) float smem[];
    const int slot = threadIdx.x, i = blockIdx.x * S + slot;  // n is a multiple of 32
    img += (size_t)i * PIX;
    w += (size_t)i * PIX;
    general_roi<R, KIND>(pix + (size_t)i * PIX, sigma[i], img, w);
    for (int k = 0; k < PIX; ++k) {
        float *q = smem + PairPixels<R>::value(k, slot, S);
        q[0] = img[k].x;
        q[PairPixels<R>::log_off(k)] = img[k].y;
    }
    float *mask = smem + 2 * PIX * S + (FULL ? slot : 4 * slot);
    if constexpr (FULL)
        for (int k = 0; k < PIX; ++k) mask[k * S] = w[k];
    else
        wle_weights_unique<R, A::MASK>(reinterpret_cast<float4 *>(mask), S, sigma[i], sigma[i], 1);
    __syncwarp();
    const PairEval<R, KIND, A::DIST, FULL> ev(smem, mask, slot, S);
    float v[P], grad[P];
    for (int k = 0; k < P; ++k) v[k] = x[(size_t)i * P + k];
    float *o = fast + (size_t)i * OUT, *g = general + (size_t)i * OUT;
    ev.gradient(v, grad);
    for (int k = 0; k < P; ++k) o[1 + k] = grad[k];
    const RoiRef roi{img, w, 1};
    numerical_gradient<R, KIND>(roi, v, g + 1);
    o[0] = ev.loss(v);  // clamps v, as loss() does
    path[i] = __all_sync(0xffffffffu, flush_safe<R, KIND>(v));
    g[0] = loss<R, KIND>(roi, v);
}

struct Buffers {
    void *p[9] = {};
    cudaError_t e = cudaSuccess;
    int n = 0;
    template <class T>
    T *get(size_t count, const T *host = nullptr) {
        T *d = nullptr;
        if (e == cudaSuccess) e = cudaMalloc(&d, count * sizeof(T));
        if (e == cudaSuccess) p[n++] = d;
        if (e == cudaSuccess && host) e = cudaMemcpy(d, host, count * sizeof(T), cudaMemcpyHostToDevice);
        return d;
    }
    ~Buffers() {
        while (n > 0) cudaFree(p[--n]);
    }
};

// G: lanes per ROI, or 1 for PairEval.
template <int R, int KIND, int G>
int run(int n, const float *pix, const float *sigma, const float *x, const float *d, float *fast, float *general,
        int *path) {
    enum { P = KindTraits<KIND>::P, PIX = R * R, OUT = (G > 1 ? 4 : 1) + P };
    if (n <= 0 || n % 32) return -1;
    Buffers b;
    const float *dp = b.get((size_t)n * PIX, pix), *ds = b.get((size_t)n, sigma), *dx = b.get((size_t)n * P, x),
                *dd = b.get((size_t)n * P, d);
    float2 *img = b.get<float2>((size_t)n * PIX);
    float *w = b.get<float>((size_t)n * PIX), *df = b.get<float>((size_t)n * OUT), *dg = b.get<float>((size_t)n * OUT);
    int *dpath = b.get<int>((size_t)n);
    if (b.e == cudaSuccess) {
        if constexpr (G > 1) {
            typedef LaneLayout<R, KIND> L;
            const int smem = (2 * L::PIXP + 32 / G * L::TOTAL) * (int)sizeof(float);
            b.e = cudaFuncSetAttribute(lanes_kernel<R, KIND, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (b.e == cudaSuccess)
                lanes_kernel<R, KIND, G><<<n / (32 / G), 32, smem>>>(n, dp, ds, dx, dd, img, w, df, dg, dpath);
        } else {
            const int smem = (2 * PIX + MaskShape<R, kFullMask<R, KIND>>::FLOATS) * 32 * (int)sizeof(float);
            b.e = cudaFuncSetAttribute(pairs_kernel<R, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (b.e == cudaSuccess) pairs_kernel<R, KIND><<<n / 32, 32, smem>>>(n, dp, ds, dx, img, w, df, dg, dpath);
        }
    }
    if (b.e == cudaSuccess) b.e = cudaGetLastError();
    if (b.e == cudaSuccess) b.e = cudaMemcpy(fast, df, (size_t)n * OUT * sizeof(float), cudaMemcpyDeviceToHost);
    if (b.e == cudaSuccess) b.e = cudaMemcpy(general, dg, (size_t)n * OUT * sizeof(float), cudaMemcpyDeviceToHost);
    if (b.e == cudaSuccess) b.e = cudaMemcpy(path, dpath, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost);
    return (int)b.e;
}

}  // namespace

extern "C" int check_exp_log(unsigned long long *out4) {
    Buffers b;
    unsigned long long *d = b.get<unsigned long long>(4);
    if (b.e == cudaSuccess) b.e = cudaMemset(d, 0, 4 * sizeof(*d));
    if (b.e == cudaSuccess) exp_log_kernel<<<148 * 8, 256>>>(d);
    if (b.e == cudaSuccess) b.e = cudaGetLastError();
    if (b.e == cudaSuccess) b.e = cudaMemcpy(out4, d, 4 * sizeof(*d), cudaMemcpyDeviceToHost);
    return (int)b.e;
}

extern "C" int check_evaluator(int R, int kind, int lanes, int n, const float *pix, const float *sigma, const float *x,
                               const float *d, float *fast, float *general, int *path) {
#define CASE(RR, KIND, G) \
    if (R == RR && kind == KIND && lanes == G) return run<RR, KIND, G>(n, pix, sigma, x, d, fast, general, path);
#define SINGLE(RR, KIND) CASE(RR, KIND, 1) CASE(RR, KIND, 16) CASE(RR, KIND, 32)
    SINGLE(7, kGS2D)
    SINGLE(9, kGS2D)
    SINGLE(11, kGS2D)
    SINGLE(13, kGS2D)
    SINGLE(7, kAS3D)
    SINGLE(9, kAS3D)
    SINGLE(11, kAS3D)
    CASE(7, k2E, 16)
    CASE(7, k2E, 32)
    CASE(11, k2E, 32)
    CASE(7, k3E, 16)
    CASE(7, k3E, 32)
    CASE(11, k3E, 32)
    CASE(7, kAS3D2E, 16)
    CASE(7, kAS3D2E, 32)
    return -1;
}
