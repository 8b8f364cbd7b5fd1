"""Value space in global memory (level 28): captured graphs beside calls of other sizes (GPU)."""

import numpy as np
import pytest
import torch

from conftest import potential_path
from mtp_b200.engine import MTPEngine

pytestmark = pytest.mark.gpu
L28 = potential_path("cfg4_L28_S4.mtp")


def _rows(n, stride=12):
    rng = np.random.default_rng(n)
    r = rng.normal(size=(n, stride, 3))
    r *= (rng.uniform(2.2, 5.2, (n, stride)) / np.linalg.norm(r, axis=-1))[..., None]
    rows = (rng.integers(0, 4, n).astype(np.int32), r, rng.integers(0, n, (n, stride)).astype(np.int32),
            rng.integers(0, 4, (n, stride)).astype(np.int32), np.full(n, stride, dtype=np.int32))
    return [torch.as_tensor(a, device="cuda") for a in rows]


def _captured(eng, rows):
    out = [torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(rows[1][:, 0]),
           torch.zeros(6, dtype=torch.float64, device="cuda")]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        eng.compute_device(*rows, energy=out[0], forces=out[1], virial=out[2])
    return g, out


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_captured_graph_beside_another_size():
    """400 atoms take one atom per block, 256 two, which need more value spaces:
    the captured graph's are still where they were."""
    a, b = _rows(400), _rows(256)
    with MTPEngine(L28, 400, 12) as eng:
        want = [t.clone() for t in eng.compute_device(*a)]
        g, out = _captured(eng, a)
        free = _free()
        eng.compute_device(*b)                  # uploads the other shape's programs (9 MB) ...
        assert free - _free() < 32 << 20        # ... and takes no other value spaces (41 MB more)
        g.replay()
        torch.cuda.synchronize()
        eng.sync_status()
        for x, y in zip(out, want):
            assert torch.equal(x, y)
        del g


def test_capture_of_one_atom_per_block_after_two():
    rows, big = _rows(100), _rows(4000)
    with MTPEngine(L28, 4000, 12) as eng:
        eng.compute_device(*big)
        assert eng.launch()["atoms_per_block"] == 2
        g, out = _captured(eng, rows)
        assert eng.launch()["atoms_per_block"] == 2
        g.replay()
        torch.cuda.synchronize()
        eng.sync_status()
        want = eng.compute_device(*rows)
        assert eng.launch()["atoms_per_block"] == 1
        for x, y in zip(out, want):
            assert (x - y).abs().max() <= 1e-10 * y.abs().max()
        del g
