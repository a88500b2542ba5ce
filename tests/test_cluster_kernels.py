"""Kernels that store into another CTA's shared memory: the CTA must be known to run first."""
import glob
import os
import re

import numpy as np
import pytest

import tp3

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "threephotons.jl_gb300", "csrc")


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            for body in f.read().split("__global__")[1:]:
                if "mapa.shared::cluster" in body:
                    yield os.path.basename(path) + ":" + re.search(r"\b(k_\w+)\(", body).group(1), body


def test_remote_stores_wait_for_the_cluster_to_run():
    """Between two cluster barriers: every CTA arrives as it starts, waits before its first remote
    store, and meets the others after it."""
    found = dict(_kernels())
    assert {"kernels_lane.cu:k_gather_lane", "kernels_tc.cu:k_finalize_parts"} <= set(found)
    for name, body in found.items():
        store = body.index("mapa.shared::cluster")
        arrive, wait, sync = (body.find(f + "();") for f in ("cluster_started_arrive", "cluster_wait", "cluster_sync"))
        assert 0 <= arrive < wait < store < sync, name
        assert body.find("__syncthreads") > arrive, name


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1, 4, 5, 8, 31, 33])
def test_idle_ctas_of_a_cluster(K):
    """Shapes at which ranks of the gather's cluster hold no shells (K < 29, K = 33) and ranks of the
    energies' sum no terms (fewer than 225 shell triples): small batches, summed by clusters, give the
    bits of batches of 160, summed by one CTA, over repeated calls."""
    L, LMAX, N = 4, 5, 4
    b = tp3.calculate_basis(L, LMAX, N, K)
    rng = np.random.default_rng(K)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = rng.normal(size=(160, K, LMAX * LMAX)) + 1j * rng.normal(size=(160, K, LMAX * LMAX))
    E = b.energy_batch(c)
    assert np.isfinite(E).all()
    for i in range(40):
        assert np.array_equal(b.energy_batch(c[4 * i:4 * i + 4]), E[4 * i:4 * i + 4])
    b.close()
