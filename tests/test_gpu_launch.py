"""The evaluation's launch shape follows the number of atoms (GPU).

Sizes at the edges of the rule's rounds (one block per SM, all resident
blocks, one more), each against the C++ FP64 oracle at the drop-in bar, and a
graph capture of a size whose shape has not been uploaded."""

import numpy as np
import pytest
import torch

from conftest import potential_path
from mtp_b200.engine import MTPEngine
from mtp_b200.mtp_file import read_mtp
from oracle.cpu_ref import CpuMTP

pytestmark = pytest.mark.gpu
NAME = "cfg1_L16_S2.mtp"


def _rows(n, stride=12):
    rng = np.random.default_rng(n)
    r = rng.normal(size=(n, stride, 3))
    r *= (rng.uniform(2.2, 4.8, (n, stride)) / np.linalg.norm(r, axis=-1))[..., None]
    return (rng.integers(0, 2, n).astype(np.int32), r, rng.integers(0, n, (n, stride)).astype(np.int32),
            rng.integers(0, 2, (n, stride)).astype(np.int32), np.full(n, stride, dtype=np.int32))


@pytest.mark.parametrize("n", [1, 2, 148, 149, 592, 593, 1185, 2369])
def test_sizes_at_the_edges_of_rounds(n):
    pot = read_mtp(potential_path(NAME))
    rows = _rows(n)
    ref = CpuMTP(pot).compute(*rows)
    with MTPEngine(potential_path(NAME), n, 12) as eng:
        out = eng.compute(*rows)
        launch = eng.launch()
    assert launch["threads"] in (128, 256, 512) and launch["atoms_per_block"] in (1, 2)
    for key in ("site_energies", "forces", "virial"):
        assert np.abs(out[key] - ref[key]).max() <= 1e-10 * np.abs(ref[key]).max(), key


@pytest.mark.parametrize("n,apb", [(148, 1), (149, 2), (297, 1), (592, 2)])
def test_value_space_in_global_memory(n, apb):
    """Level 28 in FP64 does not fit in shared memory; one or two atoms share a
    block by the number of rounds.  (148 SMs.)"""
    name = "cfg4_L28_S4.mtp"
    pot = read_mtp(potential_path(name))
    rows = _rows(n)
    ref = CpuMTP(pot).compute(*rows)
    with MTPEngine(potential_path(name), n, 12) as eng:
        out = eng.compute(*rows)
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert eng.launch()["atoms_per_block"] == apb
    for key in ("site_energies", "forces", "virial"):
        assert np.abs(out[key] - ref[key]).max() <= 1e-10 * np.abs(ref[key]).max(), key


@pytest.mark.parametrize("n,stride,hub", [(1023, 4, False), (1025, 4, False), (8192, 3, False), (8193, 3, False),
                                          (90, 12, True)])
def test_incoming_lists(n, stride, hub):
    """Sizes around the one-block scan's limits; with `hub` every slot points at
    atom 0, a list too long to sort in registers."""
    pot = read_mtp(potential_path(NAME))
    it, r, js, jt, counts = _rows(n, stride)
    if hub:
        js[:] = 0
    js[::7, 1] = n + 3                       # a neighbour without an owner: no reaction force
    ref = CpuMTP(pot).compute(it, r, js, jt, counts)
    with MTPEngine(potential_path(NAME), n, stride) as eng:
        out = eng.compute(it, r, js, jt, counts)
        again = eng.compute(it, r, js, jt, counts)
    assert np.abs(out["forces"] - ref["forces"]).max() <= 1e-10 * np.abs(ref["forces"]).max()
    assert np.array_equal(out["forces"], again["forces"])
    assert abs(out["energy"] - ref["energy"]) <= 1e-10 * abs(ref["energy"])


def test_capture_of_another_size():
    big, small = 2000, 100
    dev = torch.device("cuda")
    put = lambda rows: [torch.as_tensor(a, device=dev) for a in rows]
    b, s = put(_rows(big)), put(_rows(small))
    path = potential_path(NAME)
    with MTPEngine(path, big, 12) as fresh:
        want = [t.clone() for t in fresh.compute_device(*s)]
        torch.cuda.synchronize()
    with MTPEngine(path, big, 12) as eng:
        eng.compute_device(*b)
        torch.cuda.synchronize()
        out = [torch.empty_like(t) for t in want]
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            eng.compute_device(*s, energy=out[0], forces=out[1], virial=out[2])
        g.replay()
        torch.cuda.synchronize()
        eng.sync_status()
        for x, y in zip(out, want):
            assert (x - y).abs().max() <= 1e-10 * y.abs().max()
        del g
