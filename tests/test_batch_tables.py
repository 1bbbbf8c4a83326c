"""Batches whose solves have tables of very different sizes: the launch's shared
memory covers what every solve lays out for itself (CPU, from the kernels'
header), and FP64 batches with small tables, tables that nearly fill shared
memory and tables read from L1 equal the oracle bit for bit in any order (GPU)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import helpers

CSRC = os.path.join(helpers.PKG, "pefdtd", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "pe_kernels.cuh"
#include "pe_kernels_tiled.cuh"
#include "pe_kernels_tma.cuh"
template <typename T> int check(const std::vector<int> &n)
{
    const size_t s = pe::batch_tma_smem(pe::stress_tma_smem<T>, n.data(), (int)n.size());
    const size_t v = pe::batch_tma_smem(pe::velocity_tma_smem<T>, n.data(), (int)n.size());
    size_t most_s = 0, most_v = 0;
    for (int k : n) {
        if (pe::stress_tma_smem<T>(k) > s || pe::velocity_tma_smem<T>(k) > v) return 1;
        most_s = most_s > pe::stress_tma_smem<T>(k) ? most_s : pe::stress_tma_smem<T>(k);
        most_v = most_v > pe::velocity_tma_smem<T>(k) ? most_v : pe::velocity_tma_smem<T>(k);
    }
    return s != most_s || v != most_v;   // and no more than that
}
int main()
{
    const int sizes[] = {1, 2, 20, 150, 179, 180, 181, 300, 511, 512, 513, 1000, 16382};
    for (int a : sizes)
        for (int b : sizes)
            for (int c : sizes)
                if (check<float>({a, b, c}) || check<double>({a, b, c})) {
                    printf("%d %d %d\n", a, b, c);
                    return 1;
                }
    return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_batch_launch_covers_every_solve(tmp_path):
    src = tmp_path / "t.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-o", exe,
                           str(src)])
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("order", [(0, 1, 2), (2, 1, 0), (1, 2, 0), (2, 0, 1)])
def test_f64_batch_of_unequal_tables(order):
    from helpers import make_small, oracle_prob
    from oracle import oracle as O
    from pefdtd import batch
    probs = [make_small(nt=40, shape=(14, 36, 40), n_grains=n - 1, sponge=2, seed=41 + n) for n in (20, 150, 300)]
    assert [len(p["rho_t"]) for p in probs] == [20, 150, 300]
    probs = [probs[i] for i in order]
    b = batch.BatchSolver([batch.spec_from_problem(p) for p in probs], dtype="float64", chunk_steps=16)
    b.run(0, 40)
    got = b.traces_numpy(40)
    b.close()
    for p, tr in zip(probs, got):
        ref = O.run_oracle(oracle_prob(p, record=p["record"], damped_record=True, dtype=np.float64),
                           dtype=np.float64, fma_mode=1)
        assert np.abs(ref).max() > 0
        assert np.array_equal(tr, ref)
