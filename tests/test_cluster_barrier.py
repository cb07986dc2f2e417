"""Cluster barriers (clu_dev.cuh): .aligned ones need the whole warp together, which the cluster
kernels do not give them; and what the plain ones are there for, a solve whose waits run out."""
import os
import re

import numpy as np
import pytest

from pyom2_b200 import _abi, build, synth
from pyom2_b200.external import ExternalMode
from pyom2_b200.model import ModelState


def test_no_aligned_cluster_barrier_in_the_sources():
    for path in build.sources() + build.headers():
        for line in open(path):
            code = line.split("//")[0]
            assert not re.search(r"barrier\.cluster\.[a-z.]*aligned", code), (os.path.basename(path), line)


# a block alone in its cluster, and several
@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(20, 16), (97, 83)])
def test_timeout_in_a_cluster_leaves_the_context_usable(nx, ny):
    M = ModelState(nx, ny, 1, enable_cyclic_x=True, coord_degree=False)
    M.dxt[2:nx + 2], M.dyt[2:ny + 2], M.dzt[:] = 2e4, 2.5e4, 4000.0
    synth.calc_grid(M)
    M.kbot[2:nx + 2, 2:ny + 2] = 1
    synth.calc_topo(M)
    forc = np.zeros(M.shape2d, order="F")
    forc[2:-2, 2:-2] = 1e-12 * np.random.default_rng(nx).standard_normal((nx, ny))
    E = ExternalMode(M)
    want = np.zeros(M.shape2d, order="F")
    ok = E.solve_rtol(forc, want, rtol=1e-10)
    assert ok["status"] == 0
    E.set_sync_timeout(0.2)
    E.inject_barrier_stall(True)
    with pytest.raises(_abi.PyOMGPUError) as e:
        E.congrad_streamfunction(forc, np.zeros(M.shape2d, order="F"))
    assert e.value.code == _abi.TIMEOUT
    got = np.zeros(M.shape2d, order="F")
    info = E.solve_rtol(forc, got, rtol=1e-10)
    assert info["status"] == 0 and info["iterations"] == ok["iterations"]
    assert np.array_equal(got, want)
