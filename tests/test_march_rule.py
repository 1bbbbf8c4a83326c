"""The planes per z-march that the host picks (pe_march.cuh, CPU): kernels with
one block per slot run in whole waves and take the least number of planes;
the pair kernels' choices, by measured times, are as good as those of whole
waves on grids where another reading of the waves was slower."""
import os
import shutil
import subprocess

import pytest

import helpers

CSRC = os.path.join(helpers.PKG, "pefdtd", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
PROGRAM = r"""
#include <cstdio>
#include "pe_march.cuh"
int main()
{
    int nz, slots, model;
    long long tiles;
    double startup;
    const pe::MarchModel *m[] = {nullptr, &pe::STRESS_PAIR_MARCH, &pe::VELOCITY_PAIR_MARCH};
    while (scanf("%d %lld %d %lf %d", &nz, &tiles, &slots, &startup, &model) == 5)
        printf("%d\n", pe::pick_zchunk(nz, tiles, slots, 148, startup, m[model]));
    return 0;
}
"""

# us of the profiled kernel by planes per march, from the lengths that whole
# waves prefer and around: (grid, model, {planes: us})
MEASURED = [((114, 48, 48), 1, {4: 23.5, 6: 23.0, 7: 24.5}), ((118, 56, 56), 1, {4: 23.9, 7: 24.8}),
            ((30, 200, 200), 1, {6: 48.4, 15: 54.2}), ((20, 24, 28), 1, {1: 13.5, 4: 19.8}),
            ((47, 120, 120), 2, {3: 24.1, 5: 20.6, 6: 22.6}), ((118, 56, 56), 2, {2: 19.7, 4: 18.3}),
            ((96, 160, 160), 2, {9: 47.5, 20: 53.2}), ((20, 24, 28), 2, {1: 10.3, 4: 14.7}),
            ((61, 83, 117), 2, {3: 23.2, 5: 20.5, 6: 22.6})]


@pytest.fixture(scope="module")
def pick(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("march")
    (d / "t.cu").write_text(PROGRAM)
    subprocess.check_call([NVCC, "-std=c++17", "-I", CSRC, "-o", str(d / "t"), str(d / "t.cu")])

    def run(rows):
        text = "\n".join(" ".join(str(v) for v in r) for r in rows)
        out = subprocess.run([str(d / "t")], input=text, capture_output=True, text=True, check=True)
        return [int(v) for v in out.stdout.split()]
    return run


def test_whole_waves_take_the_least_planes(pick):
    rows = [(nz, t, 148, s, 0) for nz in (1, 7, 20, 61, 84, 136, 170) for t in (1, 9, 72, 78, 150, 400) for s in (3, 4)]
    for (nz, t, slots, s, _), zc in zip(rows, pick(rows)):
        cost = {z: -(-t * -(-nz // z) // slots) * (z + s) for z in range(1, nz + 1)}
        assert cost[zc] == min(cost.values()), (nz, t, zc)


def whole_waves(nz, tiles, slots, startup, least):
    """The march of at least `least` planes that takes the least whole waves x planes (the longest such)."""
    lengths = [z for z in sorted({-(-nz // n) for n in range(1, nz + 1)}, reverse=True) if z >= least] or [nz]
    return min(lengths, key=lambda z: -(-tiles * -(-nz // z) // slots) * (z + startup))


def test_pair_choices_lose_nothing_against_whole_waves(pick):
    rows = []
    for (nz, ny, nx), model, _ in MEASURED:
        tiles = ((nx + 30) // 30) * ((ny + 13) // 14) if model == 1 else ((nx + 31) // 32) * ((ny + 15) // 16)
        rows.append((nz, tiles, 296, 0, model))
    for (nz, tiles, slots, _, model), (grid, _, us), zc in zip(rows, MEASURED, pick(rows)):
        assert us[zc] <= 1.004 * us[whole_waves(nz, tiles, slots, 4 - model, 4)], (grid, model, zc)
