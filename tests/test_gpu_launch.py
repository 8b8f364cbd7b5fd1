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
