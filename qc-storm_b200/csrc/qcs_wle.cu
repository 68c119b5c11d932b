// WLE pre-pass (weighted-MLE parameters) over a batch of ROI records:
//   widths_keys_kernel row/column means -> natural cubic spline x10 -> peak ->
//                      two-sided widths sigma L/R/U/D, neighbour keys
//                      (WLEParaEstimation_core.h:44-156, SplineInterpolation.h:40-202,
//                      WLEParaEstimation_core.cu:21-28, 91-136)
//   nearest neighbour  same-frame minimum centre distance
//                      (WLEParaEstimation_core.cu:140-183)
//   molecule type      MLEFit / WLEFit / MultiFit
//                      (WLEParaEstimation_core.cu:197-264)
// The floating-point code keeps the reference's expression shapes (bit-equal
// results).  The nearest-neighbour search replaces the reference's O(N^2)
// all-pairs loop with a (frame, y, x) radix sort and a y-bounded scan of the
// sorted neighbours; the integer squared distance it minimises is the same.
// Records produced by ROI extraction are already in (frame, y, x) order;
// launch_wle_presorted takes their range from device memory and scans their
// compact key array without the sort, so the pass needs no host
// synchronisation.
#include <cstdint>
#include <cub/device/device_radix_sort.cuh>
#include <cuda_runtime.h>

#include "qcs_kernels.h"

namespace qcs {
namespace {

constexpr int kInterp = 10;                    // InterpolationRatio
#define QCS_INTERP_GAP (1.0f / kInterp)        // InterpolationGap
#define QCS_PEAK_FIND_RATIO 0.8f               // PeakFindRangeRatio
#define QCS_MAX_WIDTH_DIFF 0.40f               // MaxTolerablePSFWidthDiff

// Records [begin, begin + n): from the arguments, or from span[0], span[1]
// in device memory when span is set (grid-stride loops cover any n).
struct Span {
    int begin, n;
    const int *span;
    __device__ __forceinline__ void get(int &b, int &m) const {
        if (span) {
            b = span[0];
            m = span[1];
        } else {
            b = begin;
            m = n;
        }
    }
};

// Two-sided widths of one profile (a record's column or row sums, integers).
// The natural cubic spline through the R means has unit knots, so its system
// has constant coefficients (elimination factors beta, folded at compile
// time); the 10 R - 9 samples at 0.1 px are evaluated where they are used
// instead of being kept: first those near the centre for the peak, then all of
// them for the two sums, each sum adding its samples in ascending order.
// Every rounding is that of the straightforward code (arrays of samples,
// general tridiagonal solve) as nvcc contracts it, found by comparing each
// choice with it on a GPU: the same widths bit for bit.
template <int R>
struct Spline {
    enum { S = R - 1, LEN = S * kInterp + 1, MID = LEN / 2, FIND = (int)(kInterp * QCS_PEAK_FIND_RATIO) };
    float A[S], B[S], C[S], D[S];
    static __device__ __forceinline__ int seg(int i) { return i / kInterp < S ? i / kInterp : S - 1; }
    // sample i (a constant after unrolling)
    __device__ __forceinline__ float at(int i) const {
        const int g = seg(i);
        const float t = i * QCS_INTERP_GAP - (float)g;
        return __fmaf_rn(__fmul_rn(__fmul_rn(D[g], t), t), t, __fmaf_rn(__fmul_rn(C[g], t), t, __fmaf_rn(B[g], t, A[g])));
    }
};

template <int R>
__device__ __forceinline__ void profile_widths(const int (&sum)[R], float &left, float &right) {
    typedef Spline<R> Sp;
    Spline<R> sp;
    int low = sum[0];
#pragma unroll
    for (int i = 1; i < R; i++) low = min(low, sum[i]);
    float a[R], y[R], c[R];
#pragma unroll
    for (int i = 0; i < R; i++) a[i] = __fdiv_rn((float)(sum[i] - low), (float)R);
    // beta[i] of the elimination: 0, then 1 / (4 - beta[i - 1])
    float beta = 0.0f, betas[R];
    y[0] = 0.0f;
    betas[0] = 0.0f;
#pragma unroll
    for (int i = 1; i < R - 1; i++) {
        const float d1 = __fsub_rn(a[i + 1], a[i]), d0 = __fsub_rn(a[i], a[i - 1]);
        // 3 d1 - 3 d0: nvcc fuses the first product, at i = 1 and R - 3 the second (5x5: at 2 neither)
        const float b = (R == 5 && i == 2)        ? __fsub_rn(__fmul_rn(3.0f, d1), __fmul_rn(3.0f, d0))
                        : (i == 1 || i == R - 3) ? __fmaf_rn(-3.0f, d0, __fmul_rn(3.0f, d1))
                                                 : __fmaf_rn(3.0f, d1, -__fmul_rn(3.0f, d0));
        y[i] = __fdiv_rn(__fsub_rn(b, y[i - 1]), 4.0f - beta);
        beta = 1.0f / (4.0f - beta);
        betas[i] = beta;
    }
    c[R - 1] = 0.0f;
#pragma unroll
    for (int i = R - 2; i >= 0; i--) c[i] = __fmaf_rn(-betas[i], c[i + 1], y[i]);
#pragma unroll
    for (int i = 0; i < R - 1; i++) {
        sp.A[i] = a[i];
        sp.B[i] = __fmaf_rn(-(1.0f / 3.0f), __fmaf_rn(2.0f, c[i], c[i + 1]), __fsub_rn(a[i + 1], a[i]));
        sp.C[i] = c[i];
        sp.D[i] = __fdiv_rn(__fsub_rn(c[i + 1], c[i]), 3.0f);
    }
    int pos = Sp::MID;
    float peak = sp.at(Sp::MID);
#pragma unroll
    for (int i = Sp::MID - Sp::FIND; i <= Sp::MID + Sp::FIND; i++) {
        const float v = sp.at(i);
        if (v > peak) {
            peak = v;
            pos = i;
        }
    }
    const int half = min(pos, (int)Sp::LEN - pos - 1);
    const int lo = pos - half, hi = pos + half;
    float sl = 0.0f, sr = 0.0f;
#pragma unroll
    for (int i = 0; i < Sp::LEN; i++) {
        const float v = sp.at(i);
        if (i <= Sp::MID + Sp::FIND) sl = (i >= lo && i <= pos) ? __fadd_rn(sl, v) : sl;
        if (i >= Sp::MID - Sp::FIND) sr = (i >= pos && i <= hi) ? __fadd_rn(sr, v) : sr;
    }
    left = __fdiv_rn(__fdiv_rn(__fmul_rn(sl, QCS_INTERP_GAP), peak), 1.2533f);
    right = __fdiv_rn(__fdiv_rn(__fmul_rn(sr, QCS_INTERP_GAP), peak), 1.2533f);
}

// The PSF widths of a tile of kTile records, two threads a record: the tile is
// copied into shared memory (coalesced; an odd word pitch), warps 0 and 1 take
// the column sums, 2 and 3 the row sums.  Called by every thread of the block;
// the rows are complete after the next block barrier.  One thread per record with
// sample arrays in local memory took 23 / 79 / 152 us for 100,000 7x7 / 60,013
// 9x9 / 100,000 11x11 records (and 13 us for keys and types in kernels of their
// own); this takes 15 / 14 / 25 us with the keys.
constexpr int kTile = 64, kTileThreads = 2 * kTile;
template <int R>
struct Tile {
    enum { WHOLE = R * (R + 1), WORDS = WHOLE / 2, PITCH = WORDS | 1 };
    uint32_t px[kTile * PITCH];
};

template <int R, int THREADS = kTileThreads>
__device__ __forceinline__ void tile_widths(Tile<R> &tile, const uint16_t *__restrict__ rois, float *__restrict__ wle,
                                            int first, int cnt) {
    typedef Tile<R> T;
    const uint16_t *src = rois + (size_t)first * T::WHOLE;
    uint16_t *dst = reinterpret_cast<uint16_t *>(tile.px);
    if ((reinterpret_cast<uintptr_t>(src) & 3) == 0) {
        const uint32_t *s4 = reinterpret_cast<const uint32_t *>(src);
        for (int i = threadIdx.x; i < cnt * T::WORDS; i += THREADS)
            tile.px[i / T::WORDS * T::PITCH + i % T::WORDS] = __ldg(s4 + i);
    } else {
        for (int i = threadIdx.x; i < cnt * T::WHOLE; i += THREADS)
            dst[i / T::WHOLE * (2 * T::PITCH) + i % T::WHOLE] = __ldg(src + i);
    }
    __syncthreads();
    const int rec = threadIdx.x % kTile, rows = threadIdx.x / kTile;
    if (rec < cnt && rows < 2) {
        const uint16_t *p = dst + rec * (2 * T::PITCH);
        int sum[R];
#pragma unroll
        for (int i = 0; i < R; i++) sum[i] = 0;
        // sums of at most 17 x 65,535 are exact as floats, so the integers' order does not matter
        if (rows) {
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int c = 0; c < R; c++) sum[r] += p[r * R + c];
        } else {
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int c = 0; c < R; c++) sum[c] += p[r * R + c];
        }
        float left, right;
        profile_widths<R>(sum, left, right);
        float *o = wle + (size_t)(first + rec) * QCS_WLE_PARA_NUM + 1 + 2 * rows;
        o[0] = left;
        o[1] = right;
    }
}

// Sort key of a record's header h: frame (32 bits) | y (16) | x (16) of the ROI centre.
__device__ __forceinline__ unsigned long long record_key(const uint16_t *h) {
    return (((unsigned long long)h[2] + 65536ull * h[3]) << 32) | ((unsigned long long)h[1] << 16) | h[0];
}

// Distance to the nearest other ROI centre of the same frame: scans the
// (frame, y, x)-sorted keys k[0..n) outwards from a, in each direction until
// the frame changes or the row distance alone exceeds the best so far.  Keys
// are fetched 8 at a time so that their loads overlap; they are examined in
// the same order as a one-by-one scan, which stops at the same key.
__device__ __forceinline__ float nn_sorted(const unsigned long long *__restrict__ k, int a, int n) {
    const unsigned long long ka = k[a];
    const unsigned long long frame = ka >> 32;
    const int ya = (int)((ka >> 16) & 0xFFFF), xa = (int)(ka & 0xFFFF);
    float best = 100000000.0f;
    bool go = true;
    for (int b = a + 1; go && b < n; b += 8) {
        unsigned long long kb[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) kb[j] = (b + j < n) ? __ldg(k + b + j) : ~0ull;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (!go) break;
            if ((kb[j] >> 32) != frame) {
                go = false;
                break;
            }
            const int dy = (int)((kb[j] >> 16) & 0xFFFF) - ya, dx = (int)(kb[j] & 0xFFFF) - xa;
            if ((float)(dy * dy) > best) {
                go = false;
                break;
            }
            best = fminf(best, (float)(dx * dx + dy * dy));
        }
    }
    go = true;
    for (int b = a - 1; go && b >= 0; b -= 8) {
        unsigned long long kb[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) kb[j] = (b - j >= 0) ? __ldg(k + b - j) : ~0ull;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (!go) break;
            if ((kb[j] >> 32) != frame) {
                go = false;
                break;
            }
            const int dy = (int)((kb[j] >> 16) & 0xFFFF) - ya, dx = (int)(kb[j] & 0xFFFF) - xa;
            if ((float)(dy * dy) > best) {
                go = false;
                break;
            }
            best = fminf(best, (float)(dx * dx + dy * dy));
        }
    }
    return sqrtf(best);
}

__device__ __forceinline__ void classify_one(const uint16_t *__restrict__ rois, float *__restrict__ wle, int gid, int R,
                                             int whole, int LocType) {
    float MaxMeanSigmaTh;
    if (LocType == QCS_LOCTYPE_GS2D)
        MaxMeanSigmaTh = R / 2.1f / 2.35f;
    else
        MaxMeanSigmaTh = R / 1.9f / 2.35f;
    const int ROIType_Detection = rois[(size_t)gid * whole + R * R + 4];
    float *w = wle + (size_t)gid * QCS_WLE_PARA_NUM;
    const float NearestNeighborDistance = w[0];
    const float SigmaL = w[1], SigmaR = w[2], SigmaU = w[3], SigmaD = w[4];
    const float diff1 = fabsf(SigmaL - SigmaR) / fminf(SigmaL, SigmaR);
    const float diff2 = fabsf(SigmaU - SigmaD) / fminf(SigmaU, SigmaD);
    const int IsContamination = (diff1 >= QCS_MAX_WIDTH_DIFF) || (diff2 >= QCS_MAX_WIDTH_DIFF);
    const float MeanSigma = (SigmaL + SigmaR + SigmaU + SigmaD) / 4;
    int MoleculeType = QCS_MOLECULE_MLEFIT;
    if ((ROIType_Detection == QCS_ROITYPE_SINGLE) && (IsContamination == 0) && (NearestNeighborDistance >= R) &&
        (MeanSigma <= MaxMeanSigmaTh))
        MoleculeType = QCS_MOLECULE_MLEFIT;
    else if ((ROIType_Detection == QCS_ROITYPE_MULTI) || (MeanSigma > MaxMeanSigmaTh) ||
             (NearestNeighborDistance < (R / 2.0f + 1.0f)))
        MoleculeType = QCS_MOLECULE_MULTIFIT;
    else
        MoleculeType = QCS_MOLECULE_WLEFIT;
    w[5] = MoleculeType;
}

// Nearest neighbour, then molecule type, of each record, over the radix-sorted keys.
__global__ void nn_scan_kernel(const unsigned long long *__restrict__ keys, const int *__restrict__ vals, int n,
                               const uint16_t *__restrict__ rois, float *__restrict__ wle, int R, int LocType) {
    const int a = threadIdx.x + blockDim.x * blockIdx.x;
    if (a >= n) return;
    const int id = vals[a];
    wle[(size_t)id * QCS_WLE_PARA_NUM + 0] = nn_sorted(keys, a, n);
    classify_one(rois, wle, id, R, R * (R + 1), LocType);
}

// Records already in ascending (frame, y, x) order with their keys in a
// compact array: PSF widths, nearest neighbour and molecule type of each
// record in one pass.
// One thread more per record looks for the neighbour while the other two take
// the widths: a batch of frames has few tiles, so a tile's chain sets the time.
constexpr int kSortedThreads = 3 * kTile;
template <int R>
__global__ void __launch_bounds__(kSortedThreads) wle_sorted_kernel(const uint16_t *__restrict__ rois,
                                                                    const unsigned long long *__restrict__ keys, Span sp,
                                                                    float *__restrict__ wle, int LocType) {
    __shared__ Tile<R> tile;
    int b0, n;
    sp.get(b0, n);
    for (int a0 = blockIdx.x * kTile; a0 < n; a0 += gridDim.x * kTile) {
        const int cnt = min(kTile, n - a0);
        tile_widths<R, kSortedThreads>(tile, rois, wle, b0 + a0, cnt);
        const int k = (int)threadIdx.x - 2 * kTile;
        if (k >= 0 && k < cnt) wle[(size_t)(b0 + a0 + k) * QCS_WLE_PARA_NUM + 0] = nn_sorted(keys + b0, a0 + k, n);
        __syncthreads();  // the tile's widths and distances are written, its pixels free
        if (threadIdx.x < cnt) classify_one(rois, wle, b0 + a0 + threadIdx.x, R, R * (R + 1), LocType);
    }
}

// PSF widths of the records, and their neighbour keys: keys[i], vals[i] = i;
// unsorted[0] = call (another number than the earlier calls', so that nothing
// has to be cleared) when some record's key is below its predecessor's,
// unsorted[1] = n, unsorted[2] = call (unsorted may be null).
template <int R>
__global__ void __launch_bounds__(kTileThreads) widths_keys_kernel(const uint16_t *__restrict__ rois, int n,
                                                                   float *__restrict__ wle,
                                                                   unsigned long long *__restrict__ keys,
                                                                   int *__restrict__ vals, int *__restrict__ unsorted,
                                                                   int call) {
    __shared__ Tile<R> tile;
    if (unsorted && blockIdx.x == 0 && threadIdx.x == 0) {
        unsorted[1] = n;
        unsorted[2] = call;
    }
    const int first = blockIdx.x * kTile, cnt = min(kTile, n - first);
    tile_widths<R>(tile, rois, wle, first, cnt);
    if (threadIdx.x < kTile) {  // two whole warps
        bool bad = false;
        if (threadIdx.x < cnt) {
            const int i = first + threadIdx.x;
            const unsigned long long k = record_key(rois + (size_t)i * Tile<R>::WHOLE + R * R);
            bad = i > 0 && record_key(rois + (size_t)(i - 1) * Tile<R>::WHOLE + R * R) > k;
            keys[i] = k;
            vals[i] = i;
        }
        if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0 && unsorted) unsorted[0] = call;
    }
}

cudaError_t launch_widths_keys(int R, const uint16_t *rois, int n, float *wle, unsigned long long *keys, int *vals,
                               int *unsorted, int call, cudaStream_t s) {
    const int grid = (n + kTile - 1) / kTile;
#define QCS_WIDTHS(RR) \
    case RR: widths_keys_kernel<RR><<<grid, kTileThreads, 0, s>>>(rois, n, wle, keys, vals, unsorted, call); break;
    switch (R) {
        QCS_WIDTHS(5)
        QCS_WIDTHS(7)
        QCS_WIDTHS(9)
        QCS_WIDTHS(11)
        QCS_WIDTHS(13)
        QCS_WIDTHS(15)
        QCS_WIDTHS(17)
    default: return cudaErrorInvalidValue;
    }
#undef QCS_WIDTHS
    return cudaGetLastError();
}

size_t sort_temp_bytes(int n) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned long long *)nullptr, (unsigned long long *)nullptr,
                                    (const int *)nullptr, (int *)nullptr, n);
    return bytes;
}

inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace

size_t wle_scratch_bytes(int n) {
    const size_t nn = (size_t)(n > 0 ? n : 1);
    return 2 * align256(nn * 8) + 2 * align256(nn * 4) + align256(sort_temp_bytes((int)nn)) + align256(3 * sizeof(int));
}

cudaError_t launch_wle(const uint16_t *rois, int n, int R, int loc_type, float *wle, void *scratch, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const size_t nn = (size_t)n;
    char *p = static_cast<char *>(scratch);
    unsigned long long *k_in = reinterpret_cast<unsigned long long *>(p);
    p += align256(nn * 8);
    unsigned long long *k_out = reinterpret_cast<unsigned long long *>(p);
    p += align256(nn * 8);
    int *v_in = reinterpret_cast<int *>(p);
    p += align256(nn * 4);
    int *v_out = reinterpret_cast<int *>(p);
    p += align256(nn * 4);
    size_t temp = sort_temp_bytes(n);
    cudaError_t e = launch_widths_keys(R, rois, n, wle, k_in, v_in, nullptr, 0, s);
    if (e != cudaSuccess) return e;
    e = cub::DeviceRadixSort::SortPairs(p, temp, k_in, k_out, v_in, v_out, n, 0, 64, s);
    if (e != cudaSuccess) return e;
    const int tpb = 64;
    nn_scan_kernel<<<(n + tpb - 1) / tpb, tpb, 0, s>>>(k_out, v_out, n, rois, wle, R, loc_type);
    return cudaGetLastError();
}

namespace {

// Fills keys[*count .. cap) with padding (all ones, after every real key).
__global__ void pad_keys_kernel(unsigned long long *__restrict__ keys, int *__restrict__ vals,
                                const int *__restrict__ count, int cap) {
    const int i = threadIdx.x + blockDim.x * blockIdx.x;
    if (i < *count || i >= cap) return;
    keys[i] = ~0ull;
    vals[i] = i;
}

// The sort of up to kSmallSort keys, by key and then index (the radix sort's
// order), in one block's shared memory; returns at once for records in order.
// Against the graph's launch: 300 records in order 23.8 -> 15.2 us, out of order
// 43 -> 23; 4,096 out of order 105 -> 70.  More keys than this do not fit one
// block's static shared memory.
constexpr int kSmallSort = 4096, kSmallThreads = 1024;
__global__ void __launch_bounds__(kSmallThreads) small_sort_kernel(const unsigned long long *__restrict__ k_in,
                                                                   unsigned long long *__restrict__ k_out,
                                                                   int *__restrict__ v_out,
                                                                   const int *__restrict__ unsorted, int n) {
    __shared__ unsigned long long key[kSmallSort];
    __shared__ int val[kSmallSort];
    if (unsorted[0] != unsorted[2]) return;
    int m = 2;
    while (m < n) m <<= 1;
    for (int i = threadIdx.x; i < m; i += kSmallThreads) {
        key[i] = i < n ? k_in[i] : ~0ull;
        val[i] = i;
    }
    __syncthreads();
    for (int k = 2; k <= m; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < m / 2; i += kSmallThreads) {
                const int a = ((i & ~(j - 1)) << 1) | (i & (j - 1)), b = a + j;
                const unsigned long long ka = key[a], kb = key[b];
                const int va = val[a], vb = val[b];
                const bool above = ka > kb || (ka == kb && va > vb);
                if (above == ((a & k) == 0)) {
                    key[a] = kb, key[b] = ka;
                    val[a] = vb, val[b] = va;
                }
            }
            __syncthreads();
        }
    for (int i = threadIdx.x; i < n; i += kSmallThreads) {
        k_out[i] = key[i];
        v_out[i] = val[i];
    }
}

// Sets the sort's IF condition from the flag of widths_keys_kernel.
__global__ void wle_sort_cond_kernel(cudaGraphConditionalHandle h, const int *__restrict__ unsorted) {
    cudaGraphSetConditional(h, unsorted[0] == unsorted[2] ? 1u : 0u);
}

// nn_scan_kernel over the sorted keys when the records were out of order,
// else over the records' own keys (already sorted, identity order).
__global__ void nn_scan_select_kernel(const unsigned long long *__restrict__ k_in, const unsigned long long *__restrict__ k_out,
                                      const int *__restrict__ v_out, const int *__restrict__ unsorted, int n,
                                      const uint16_t *__restrict__ rois, float *__restrict__ wle, int R, int LocType) {
    const int a = threadIdx.x + blockDim.x * blockIdx.x;
    if (a >= n) return;
    const bool sorted = unsorted[0] != unsorted[2];
    const int id = sorted ? a : v_out[a];
    wle[(size_t)id * QCS_WLE_PARA_NUM + 0] = nn_sorted(sorted ? k_in : k_out, a, n);
    classify_one(rois, wle, id, R, R * (R + 1), LocType);
}

}  // namespace

// The WLE pre-pass of a localization context.  Records produced by ROI
// extraction (and most callers' batches) are already in (frame, y, x)
// order; then the radix sort of the nearest-neighbour keys is the identity
// and only costs time.  Here widths_keys_kernel flags out-of-order records and
// a CUDA graph holds the sort inside an IF node whose condition a one-thread
// kernel sets from that flag, so the sort runs only when needed and the host
// never waits.  The sort covers `capacity` keys (padded inside the node); up to
// kSmallSort keys have a launch of their own instead.
struct WleSorter {
    int capacity = 0;
    void *scratch = nullptr;  // wle_scratch_bytes(capacity), owned by the caller
    unsigned long long *k_in = nullptr, *k_out = nullptr;
    int *v_in = nullptr, *v_out = nullptr, *flag = nullptr;
    int call = 0;  // the last call's number (widths_keys_kernel)
    cudaStream_t cap = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

void wle_sorter_destroy(WleSorter *w) {
    if (!w) return;
    if (w->exec) cudaGraphExecDestroy(w->exec);
    if (w->graph) cudaGraphDestroy(w->graph);
    if (w->cap) cudaStreamDestroy(w->cap);
    delete w;
}

cudaError_t wle_sorter_create(int capacity, void *scratch, WleSorter **out) {
    *out = nullptr;
    WleSorter *w = new WleSorter();
    w->capacity = capacity;
    w->scratch = scratch;
    const size_t nn = (size_t)capacity;
    char *p = static_cast<char *>(scratch);
    w->k_in = reinterpret_cast<unsigned long long *>(p);
    p += align256(nn * 8);
    w->k_out = reinterpret_cast<unsigned long long *>(p);
    p += align256(nn * 8);
    w->v_in = reinterpret_cast<int *>(p);
    p += align256(nn * 4);
    w->v_out = reinterpret_cast<int *>(p);
    p += align256(nn * 4);
    void *temp = p;
    size_t temp_bytes = sort_temp_bytes(capacity);
    p += align256(temp_bytes);
    w->flag = reinterpret_cast<int *>(p);

    cudaGraphConditionalHandle h = 0;
    cudaGraphNode_t kn = nullptr, cn = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&w->cap, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemsetAsync(w->flag, 0, 3 * sizeof(int), w->cap);
    if (e == cudaSuccess) e = cudaStreamSynchronize(w->cap);  // before a call on any stream
    if (e == cudaSuccess) e = cudaGraphCreate(&w->graph, 0);
    if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&h, w->graph, 0, cudaGraphCondAssignDefault);
    if (e == cudaSuccess) {
        cudaKernelNodeParams kp = {};
        const int *flag = w->flag;
        void *args[] = {&h, &flag};
        kp.func = reinterpret_cast<void *>(wle_sort_cond_kernel);
        kp.gridDim = dim3(1);
        kp.blockDim = dim3(1);
        kp.sharedMemBytes = 0;
        kp.kernelParams = args;
        e = cudaGraphAddKernelNode(&kn, w->graph, nullptr, 0, &kp);
    }
    cudaGraph_t body = nullptr;
    if (e == cudaSuccess) {
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeIf;
        cp.conditional.size = 1;
        e = cudaGraphAddNode(&cn, w->graph, &kn, 1, &cp);
        if (e == cudaSuccess) body = cp.conditional.phGraph_out[0];
    }
    if (e == cudaSuccess)
        e = cudaStreamBeginCaptureToGraph(w->cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed);
    if (e == cudaSuccess) {
        pad_keys_kernel<<<(capacity + 255) / 256, 256, 0, w->cap>>>(w->k_in, w->v_in, w->flag + 1, capacity);
        cudaError_t es = cub::DeviceRadixSort::SortPairs(temp, temp_bytes, w->k_in, w->k_out, w->v_in, w->v_out,
                                                         capacity, 0, 64, w->cap);
        cudaGraph_t captured = nullptr;
        e = cudaStreamEndCapture(w->cap, &captured);
        if (e == cudaSuccess) e = es;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&w->exec, w->graph, 0);
    if (e != cudaSuccess) {
        cudaGetLastError();
        wle_sorter_destroy(w);
        return e;
    }
    *out = w;
    return cudaSuccess;
}

cudaError_t launch_wle_ctx(WleSorter *w, const uint16_t *rois, int n, int R, int loc_type, float *wle,
                           cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s, &cs);
    if (e != cudaSuccess) return e;
    if (n > w->capacity || cs != cudaStreamCaptureStatusNone)
        return launch_wle(rois, n, R, loc_type, wle, w->scratch, s);
    if (++w->call == 0) ++w->call;  // 0: the cleared flag's
    e = launch_widths_keys(R, rois, n, wle, w->k_in, w->v_in, w->flag, w->call, s);
    if (e != cudaSuccess) return e;
    if (n <= kSmallSort) {
        small_sort_kernel<<<1, kSmallThreads, 0, s>>>(w->k_in, w->k_out, w->v_out, w->flag, n);
        e = cudaGetLastError();
    } else {
        e = cudaGraphLaunch(w->exec, s);
    }
    if (e != cudaSuccess) return e;
    const int tpb = 64;
    nn_scan_select_kernel<<<(n + tpb - 1) / tpb, tpb, 0, s>>>(w->k_in, w->k_out, w->v_out, w->flag, n, rois, wle, R,
                                                              loc_type);
    return cudaGetLastError();
}

cudaError_t launch_wle_presorted(const uint16_t *rois, const unsigned long long *keys, const int *d_span, int max_n,
                                 int R, int loc_type, float *wle, cudaStream_t s) {
    if (max_n <= 0) return cudaSuccess;
    int grid = (max_n + kTile - 1) / kTile;
    if (grid > 148 * 8) grid = 148 * 8;
    const Span sp{0, 0, d_span};
    switch (R) {
    case 5: wle_sorted_kernel<5><<<grid, kSortedThreads, 0, s>>>(rois, keys, sp, wle, loc_type); break;
    case 7: wle_sorted_kernel<7><<<grid, kSortedThreads, 0, s>>>(rois, keys, sp, wle, loc_type); break;
    case 9: wle_sorted_kernel<9><<<grid, kSortedThreads, 0, s>>>(rois, keys, sp, wle, loc_type); break;
    case 11: wle_sorted_kernel<11><<<grid, kSortedThreads, 0, s>>>(rois, keys, sp, wle, loc_type); break;
    case 13: wle_sorted_kernel<13><<<grid, kSortedThreads, 0, s>>>(rois, keys, sp, wle, loc_type); break;
    case 15: wle_sorted_kernel<15><<<grid, kSortedThreads, 0, s>>>(rois, keys, sp, wle, loc_type); break;
    case 17: wle_sorted_kernel<17><<<grid, kSortedThreads, 0, s>>>(rois, keys, sp, wle, loc_type); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace qcs
