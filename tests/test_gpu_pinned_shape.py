"""A launch shape pinned with set_launch gives an atom the same bits in systems of any size (GPU)."""

import numpy as np
import pytest
import torch

from conftest import potential_path
from mtp_b200.engine import MTPEngine

pytestmark = pytest.mark.gpu


def _rows(n, stride=20):
    rng = np.random.default_rng(7)
    r = rng.normal(size=(n, stride, 3))
    r *= (rng.uniform(2.2, 5.5, (n, stride)) / np.linalg.norm(r, axis=-1))[..., None]   # some beyond the cutoff
    rows = (rng.integers(0, 2, n).astype(np.int32), r, np.full((n, stride), -1, dtype=np.int32),
            rng.integers(-1, 2, (n, stride)).astype(np.int32), rng.integers(0, stride + 1, n).astype(np.int32))
    return [torch.as_tensor(a, device="cuda") for a in rows]


@pytest.mark.parametrize("name,precision,threads,atoms", [("cfg3_L20_S2.mtp", "mixed", 512, 4),
                                                          ("cfg3_L20_S2.mtp", "mixed", 256, 0),
                                                          ("cfg1_L16_S2.mtp", "fp64", 128, 2),
                                                          ("cfg2_L24_S3.mtp", "mixed", 128, 2)])
def test_same_bits_for_every_size(name, precision, threads, atoms):
    rows = _rows(2400)
    with MTPEngine(potential_path(name), 2400, 20, precision=precision) as eng:
        eng.set_launch(threads, 0, atoms)
        got = {}
        for n in (3, 149, 600, 2400):
            e = torch.zeros(n, dtype=torch.float64, device="cuda")
            _, f, _ = eng.compute_device(*[t[:n] for t in rows], eatom=e)
            eng.sync_status()
            if threads and atoms:
                assert (eng.launch()["threads"], eng.launch()["atoms_per_block"]) == (threads, atoms)
            got[n] = (e, f.clone())
        for n, (e, f) in got.items():
            assert torch.equal(e, got[2400][0][:n]) and torch.equal(f, got[2400][1][:n]), n
