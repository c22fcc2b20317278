"""The host-side rules of the M <= 64 kernel (include/gemm/stacked_k_plan.h), walked over its range without a GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SMS, SMEM_PER_BLOCK, SMEM_PER_SM, SMEM_RESERVED, TMEM_COLS, THREADS_PER_SM = 148, 232448, 233472, 1024, 512, 2048

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "gemm/stacked_k_plan.h"
int main(int, char** argv) {
    const uint32_t sms = std::atoi(argv[1]), max_smem = std::atoi(argv[2]), cap = std::atoi(argv[3]);
    for (uint32_t m : {1u, 16u, 17u, 32u, 33u, 64u})
        for (uint32_t n = 16; n <= 9600; n += 16)
            for (uint32_t k = 128; k <= 18432; k += 128) {
                if (!yan::stacked_k_preferred(m, n, k, cap, sms, max_smem)) continue;
                const yan::StackedConfig c = yan::choose_stacked_config(m, n, k, cap, sms, max_smem);
                if (cap == sms && c.cluster == 1) continue;
                const uint32_t steps = yan::stacked_k_steps(k, c.stack, c.cluster);
                std::printf("%u %u %u %u %u %u %u\n", m, n, k, c.cluster, yan::ceil_div(n, 128u / c.stack) * c.cluster,
                            yan::stacked_k_smem_layout(c.m_pad, c.stack, steps, c.slots, c.cluster).total,
                            yan::stacked_k_tmem_cols(c.m_pad, c.stack, c.slots));
            }
    std::printf("threads %u\n", yan::kStackedThreads);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    assert cxx, "g++ not found: set CXX"
    d = tmp_path_factory.mktemp("plan")
    (d / "walk.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-D__host__=", "-D__device__=", f"-I{ROOT}/yan_b200/include", str(d / "walk.cpp"),
                    "-o", str(d / "walk")], check=True)

    def walk(cap):
        out = subprocess.run([str(d / "walk"), str(SMS), str(SMEM_PER_BLOCK), str(cap)], check=True, capture_output=True, text=True)
        lines = out.stdout.splitlines()
        return np.array([[int(x) for x in line.split()] for line in lines[:-1]]), int(lines[-1].split()[1])
    return walk


@pytest.fixture(scope="module")
def walk(program):
    """Rows of (M, N, K, CTAs per cluster, CTAs, shared memory, tensor-memory columns) of every configuration with a cluster."""
    rows, threads = program(SMS)
    assert len(rows) > 1000
    return rows, threads


def test_tensor_memory_of_the_ctas_that_share_an_sm(walk):
    """CTAs of clusters that fit an SM by shared memory and threads also fit by tensor memory: none waits for another's
    columns.  (Registers, which may keep a second CTA away, are left out: the bound is on the safe side.)"""
    rows, threads = walk
    per_sm = np.minimum(SMEM_PER_SM // (rows[:, 5] + SMEM_RESERVED), THREADS_PER_SM // threads)
    bad = rows[per_sm * rows[:, 6] > TMEM_COLS]
    assert len(bad) == 0, f"{len(bad)} configurations, e.g. (M, N, K, cluster, CTAs, smem, columns) = {bad[:3].tolist()}"


def test_clusters_are_resident_at_once(walk):
    """Clusters of two up to one CTA per SM; clusters of four, which not every SM can be part of, up to 132 CTAs unless two fit
    an SM."""
    rows, _ = walk
    assert set(rows[:, 3]) == {2, 4} and rows[:, 4].max() <= SMS
    one_per_sm = 2 * (rows[:, 5] + SMEM_RESERVED) > SMEM_PER_SM
    assert rows[(rows[:, 3] == 4) & one_per_sm][:, 4].max() == 132


@pytest.mark.parametrize("cap", [1, 37, 124, 147])
def test_a_cap_on_the_sms_bounds_the_grid(program, cap):
    """Where this kernel is the default under a cap it has no more CTAs, and it is the default wherever 64-row groups fit."""
    rows, _ = program(cap)
    assert rows[:, 4].max() <= cap
    fits = {(m, n, k) for m, n, k in rows[:, :3].tolist()}
    assert all((m, n, 2048) in fits for m in (1, 16, 17, 32, 64) for n in range(16, min(64 * cap, 9600) + 1, 16))
