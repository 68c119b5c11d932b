"""Workspace of the layers' weight and bias gradients (qcs_gemm_plan.h): every
layer's partial products and column sums lie inside the workspace, apart from
one another, for any workspace size; the splits cover K; and the workspace of a
network splits K as far as the SMs ask."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <algorithm>
#include <cstdio>
#include <utility>
#include <vector>
#include "qcs_gemm_plan.h"
using namespace qcs::learned;

int main() {
    long bad = 0, refused = 0, split = 0;
    const int kins[] = {64, 96, 136, 176, 232, 304}, outs[] = {8, 16}, rows[] = {0, 1, 255, 256, 512, 4096, 20000, 65536};
    const size_t sizes[] = {0, 7, 263, 264, 265, 300, 16895, 16896, 16897, 20000, 40000, 65536, 131072, 262144, 300000, 1 << 21};
    for (int kin : kins) for (int no : outs) for (int K : rows) for (int most : {0, 1, 5, 8, 16, 148}) for (size_t ws : sizes) {
        const int M[3] = {kin, 128, 128}, N[3] = {128, 128, no};
        LayerSplit p[3];
        if (!plan_layers(3, M, N, K, most, ws, p)) {
            refused++;
            bad += ws >= (size_t)(N[0] + N[1] + N[2]);
            continue;
        }
        std::vector<std::pair<size_t, size_t>> used;
        for (int i = 0; i < 3; i++) {
            const int z = p[i].split.z, kper = p[i].split.kper;
            bad += z < 1 || z > std::max(most, 1) || (long long)z * kper < K || (z > 1 && (long long)(z - 1) * kper >= K);
            if (z > 1) used.push_back({p[i].part, p[i].part + (size_t)z * M[i] * N[i]});
            used.push_back({p[i].sums, p[i].sums + (size_t)z * N[i]});
            split += z > 1;
            if (ws == (1 << 21)) bad += z != gemm_split(M[i], N[i], K, most, ws).z && most <= 16;
        }
        std::sort(used.begin(), used.end());
        for (size_t i = 0; i < used.size(); i++) bad += used[i].second > (i + 1 < used.size() ? used[i + 1].first : ws);
    }
    printf("%ld %ld %ld\n", bad, refused, split);
    return 0;
}
"""


def test_layer_splits_stay_inside_the_workspace(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "qc-storm_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    bad, refused, split = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0
    assert refused > 0 and split > 0
