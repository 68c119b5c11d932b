// How the training products divide K and their workspace (host arithmetic only).
#pragma once

#include <cstddef>

namespace qcs {
namespace learned {

constexpr int kGemmK = 128;       // depth of a K chunk
constexpr int kGemmSplits = 64;   // K ranges per tile at most

// z ranges of kper of K each (z = 1: not split).
struct GemmSplit {
    int z, kper;
};

// K over at most `most` CTAs a tile, at least 256 of K each, with z M N partial
// sums in at most ws_floats.
inline GemmSplit gemm_split(int M, int N, int K, int most, size_t ws_floats) {
    int s = most;
    const int by_k = K / 256;
    if (s > by_k) s = by_k;
    if (s > kGemmSplits) s = kGemmSplits;
    while (s > 1 && (size_t)s * M * N > ws_floats) --s;
    if (s < 1) s = 1;
    int kper = (K + s - 1) / s;
    kper = ((kper + kGemmK - 1) / kGemmK) * kGemmK;
    const int z = kper > 0 ? (K + kper - 1) / kper : 1;
    return z > 1 ? GemmSplit{z, kper} : GemmSplit{1, K};
}

// A layer's weight gradient (M x N) and bias gradient (N column sums) in one
// workspace: split z's partial products at part + z M N (where split), its column
// sums at sums + z N.
struct LayerSplit {
    GemmSplit split;
    size_t part, sums;  // floats from the workspace's start
};

// The splits of `layers` layers of K rows, `most` CTAs a tile.  Room for every
// layer's column sums is set aside before any layer's partials; where that does
// not fit, no layer is split.  False: not even one sum a column fits.
inline bool plan_layers(int layers, const int *M, const int *N, int K, int most, size_t ws_floats, LayerSplit *out) {
    size_t one = 0;
    for (int i = 0; i < layers; ++i) one += (size_t)N[i];
    if (one > ws_floats) return false;
    const bool split = one * kGemmSplits <= ws_floats;
    size_t left = split ? ws_floats - one * kGemmSplits : 0, at = 0;
    for (int i = 0; i < layers; ++i) {
        out[i].split = split ? gemm_split(M[i], N[i], K, most, left) : GemmSplit{1, K};
        const size_t part = out[i].split.z > 1 ? (size_t)out[i].split.z * M[i] * N[i] : 0;
        out[i].part = at;
        out[i].sums = at + part;
        at += part + (size_t)out[i].split.z * N[i];
        left -= part;
    }
    return true;
}

}  // namespace learned
}  // namespace qcs
