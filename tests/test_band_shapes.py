"""The unit-cost bands' choice of a window (csrc/edit.cuh), compiled by the host's compiler, against its rule restated
here step by step."""

import os
import subprocess

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(1 << (s // 6), s % 6 + 1) for s in range(36)] + [(32, 8), (32, 12), (32, 16)]

PROGRAM = r"""
#include "edit.cuh"
#include <cstdio>
int main() {
    long long n, m, t, chain;
    int latency, reach;
    dinara::BandTuning tuning = dinara::default_band_tuning();
    for (int s = 0; s < dinara::kBandShapes; ++s)
        if (std::scanf("%f", &tuning.word_cost[s]) != 1) return 1;
    while (std::scanf("%lld %lld %lld %d %lld %d", &n, &m, &t, &latency, &chain, &reach) == 6) {
        tuning.chain_words = chain;
        tuning.reach = reach;
        std::printf("%d\n", dinara::band_shape_for(n, m, t, latency != 0, tuning));
    }
}
"""


def _chosen(n, m, t, latency, chain, reach, costs):
    delta = m - n
    e = (t - delta) // 2 if t > delta else 0
    needed = min((delta + 2 * e + 1 + 63) // 64 + 1, (n + 63) // 64)
    sizes = [lanes * words for lanes, words in SHAPES]
    holding = [s for s in range(len(SHAPES)) if sizes[s] >= needed]
    if not holding:
        return len(SHAPES) - 1
    smallest = min(sizes[s] for s in holding)
    price = [np.float32(np.float32(sizes[s]) * costs[s]) for s in range(len(SHAPES))]
    if latency:
        return min((s for s in holding if sizes[s] <= 2 * smallest), key=lambda s: (SHAPES[s][1], sizes[s], s))
    for quarters in ([5] if reach >= 5 else []) + ([reach] if reach > 5 else []):
        fits = [s for s in holding if 4 * sizes[s] <= quarters * smallest and m * SHAPES[s][1] <= chain]
        if fits:
            return min(fits, key=lambda s: (price[s], s))
    within = [s for s in holding if 4 * sizes[s] <= max(reach, 5) * smallest]
    return min(within, key=lambda s: (m * SHAPES[s][1], price[s], s))


def test_choice_of_a_window(tmp_path):
    rng = np.random.default_rng(39)
    path, program = tmp_path / "shapes.cpp", tmp_path / "shapes"
    path.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "dinara-align_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include", str(path), "-o", str(program),
                    "-L", "/usr/local/cuda/lib64", "-lcudart"], check=True, capture_output=True, text=True)
    for trial in range(4):
        # Costs apart and, in the last two trials, many of them alike.
        costs = (rng.uniform(30, 60, len(SHAPES)) if trial < 2 else rng.choice([40, 50], len(SHAPES))).astype(np.float32)
        calls = []
        for _ in range(4000):
            n = int(np.exp(rng.uniform(0, np.log(60_000))))
            m = n + int(rng.choice([0, 1, 60, 64, 500, n]))
            t = int(np.exp(rng.uniform(0, np.log(n + m + 2))))
            calls.append((n, m, t, int(rng.integers(0, 2)), int(rng.choice([1000, 24_000, 48_000, 400_000])),
                          int(rng.choice([4, 5, 6, 8]))))
        text = " ".join(repr(float(c)) for c in costs) + "\n" + "\n".join(" ".join(map(str, c)) for c in calls)
        run = subprocess.run([str(program)], input=text, capture_output=True, text=True, check=True, timeout=60)
        assert [int(line) for line in run.stdout.split()] == [_chosen(*call, costs) for call in calls]
