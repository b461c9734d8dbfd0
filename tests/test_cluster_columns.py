"""Cluster launches and tensor memory: CTAs of clusters from two launches may share SMs
only while their columns fit together, since a CTA waits for columns without a limit and
for its cluster's peers at a barrier."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from filtered_tdma_b200 import Solver
from filtered_tdma_b200 import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "k_tile_any.cuh"
using namespace btdma;
// Prints "warps columns bytes" for CTAs of 1 to 16 warps that need `need` bytes.
int main() {
    const size_t sm = 233472;  // shared memory of an SM (sm_100)
    for (int warps = 1; warps <= 16; ++warps) {
        const int cols = wide_tmem_cols(warps);
        for (size_t need = 4096; need <= 232448; need += 4096)
            std::printf("%d %d %zu %zu\n", warps, cols, need, wide_cluster_smem(need, cols, sm));
    }
}
"""


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="no nvcc")
def test_resident_ctas_fit_the_columns(tmp_path):
    src = tmp_path / "columns.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "columns"
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "filtered_tdma_b200", "csrc"), "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(rows) > 500
    # any two that fit an SM together (each takes 1 KB more) fit its 512 columns, at most
    # 256 each, so that a free aligned block is left for the other; no three fit
    least = {}
    for _, cols, _, smem in rows:
        least[cols] = min(least.get(cols, 1 << 30), smem + 1024)
    for c1, b1 in least.items():
        for c2, b2 in least.items():
            assert b1 + b2 > 233472 or max(c1, c2) <= 256
    assert 3 * min(least.values()) > 233472


@pytest.mark.gpu
def test_two_streams_of_clusters(cuda, orc):
    import torch
    # 512 and 256 columns a CTA; tensor-map and cp.async forms
    shapes = [(2401, 545, False), (601, 1537, True), (602, 700, True), (2400, 1024, False)]
    jobs = []
    for n_sys, n_row, cyclic in shapes:
        arrays = W.row_varying(n_sys, n_row, seed=n_row)
        ref = orc.thomas_cyclic(*arrays) if cyclic else orc.thomas(*arrays)
        dev = [torch.from_numpy(np.ascontiguousarray(v)).to(cuda) for v in arrays]
        s = Solver("pascal", n_sys, n_row, 16)
        X = torch.empty_like(dev[3])
        s.solve_out(*dev, X, cyclic=cyclic)
        assert np.max(np.abs(X.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))
        jobs.append((s, dev, X, cyclic))
    first = [job[2].clone() for job in jobs]
    for job in jobs:
        job[2].zero_()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in jobs]
    for _ in range(20):
        for (s, dev, X, cyclic), st in zip(jobs, streams):
            with torch.cuda.stream(st):
                s.solve_out(*dev, X, cyclic=cyclic)
    torch.cuda.synchronize()
    for (s, _, X, _), want in zip(jobs, first):
        assert torch.equal(X, want)
        assert s.status() == 0
