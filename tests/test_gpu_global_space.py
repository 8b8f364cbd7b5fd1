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
        eng.compute_device(*b)                  # uploads the other shape's programs
        free = _free()
        eng.compute_device(*a)
        eng.compute_device(*b)
        assert _free() == free                  # nothing was allocated or given back
        g.replay()
        torch.cuda.synchronize()
        eng.sync_status()
        for x, y in zip(out, want):
            assert torch.equal(x, y)
        del g
