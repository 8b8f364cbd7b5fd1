"""Rows of every staging layout (GPU).

A staging row is an odd number of 16-byte words long or, where that fits another
block on an SM, just the words that its slots need; long rows end anywhere in
between.  Each shape at the edges of its range, against the C++ FP64 oracle:
1e-10 relative in FP64; in mixed precision FP32 rounding (6e-8) times the terms
of the sums (the row and about 1e3 products) times the four basic moments that a
product may have.  The coefficient gradient: 1e-8 against torch double backward."""

import numpy as np
import pytest
import torch

from conftest import potential_path
from mtp_b200.engine import MTPEngine
from mtp_b200.mtp_file import read_mtp
from mtp_b200.train import DeviceBatch, predict, weighted_loss
from oracle import mtp_oracle as O
from oracle.cpu_ref import CpuMTP

pytestmark = pytest.mark.gpu
L16, L20, L24, L28 = "cfg1_L16_S2.mtp", "cfg3_L20_S2.mtp", "cfg2_L24_S3.mtp", "cfg4_L28_S4.mtp"


def _rows(stride, n=13):
    rng = np.random.default_rng(stride)
    r = rng.normal(size=(n, stride, 3))
    r *= (rng.uniform(2.2, 5.3, (n, stride)) / np.linalg.norm(r, axis=-1))[..., None]   # some past the cutoff
    counts = np.resize([stride, 0, 1, stride // 2, stride - 1, max(0, stride - 2)], n).astype(np.int32)
    return (rng.integers(0, 2, n).astype(np.int32), r, rng.integers(0, n, (n, stride)).astype(np.int32),
            rng.integers(0, 2, (n, stride)).astype(np.int32), counts)


@pytest.mark.parametrize("name,precision,threads,atoms,stride", [
    (L24, "mixed", 512, 4, 64), (L24, "mixed", 512, 4, 69), (L24, "mixed", 512, 4, 76), (L24, "mixed", 256, 4, 84),
    (L24, "mixed", 128, 4, 88), (L24, "mixed", 256, 2, 76), (L24, "fp64", 512, 2, 64), (L24, "fp64", 512, 2, 75),
    (L24, "fp64", 512, 2, 76), (L24, "fp64", 512, 2, 78), (L24, "fp64", 256, 2, 83), (L20, "fp64", 256, 2, 105),
    (L20, "mixed", 128, 4, 12), (L20, "mixed", 256, 4, 104), (L16, "mixed", 128, 4, 81), (L16, "mixed", 128, 4, 124),
    (L16, "fp64", 128, 2, 86), (L16, "fp64", 256, 1, 257), (L16, "mixed", 512, 4, 260), (L16, "mixed", 128, 1, 1024),
    (L16, "fp64", 512, 2, 300), (L16, "fp64", 512, 1, 905), (L20, "mixed", 512, 2, 301)])
def test_rows_match_oracle(name, precision, threads, atoms, stride):
    pot = read_mtp(potential_path(name))
    rows = _rows(stride)
    ref = CpuMTP(pot).compute(*rows)
    tol = 1e-10 if precision == "fp64" else 4 * (stride + 1000) * 6e-8
    with MTPEngine(potential_path(name), len(rows[0]), stride, precision=precision) as eng:
        eng.set_launch(threads, 0, atoms)
        out = eng.compute(*rows)
        ran = eng.launch()
    assert (ran["threads"], ran["atoms_per_block"]) == (threads, atoms)
    for key in ("site_energies", "forces", "virial"):
        assert np.abs(out[key] - ref[key]).max() <= tol * np.abs(ref[key]).max(), key


@pytest.mark.parametrize("n,stride", [(13, 600), (149, 600), (297, 500)])
def test_mixed_value_space_in_global_memory(n, stride):
    """Rows too long for level 28 in shared memory also in mixed precision."""
    pot = read_mtp(potential_path(L28))
    rows = _rows(stride, n)
    with MTPEngine(potential_path(L28), n, stride, precision="mixed") as eng:
        out = eng.compute(*rows)
        assert eng.launch()["atoms_per_block"] == 1
    ref = CpuMTP(pot).compute(*rows)
    tol = 4 * (stride + 1000) * 6e-8
    for key in ("site_energies", "forces", "virial"):
        assert np.abs(out[key] - ref[key]).max() <= tol * np.abs(ref[key]).max(), key


@pytest.mark.parametrize("stride", [192, 193, 256, 257, 300])
def test_adjoint_of_long_rows(stride):
    name = "cfg3_L20_S2.mtp"
    pot = read_mtp(potential_path(name))
    it, r, js, jt, counts = _rows(stride, 7)
    N = len(it)
    jt[np.arange(stride)[None] >= counts[:, None]] = -1
    cfg = np.zeros(N, dtype=np.int32)
    vols = np.array([900.0])
    rng = np.random.default_rng(3)
    targets = (rng.normal(size=1) * 10, rng.normal(size=(N, 3)), rng.normal(size=(1, 6)) * 1e-2)
    params = {"species": pot.species_coeffs, "radial": pot.radial_coeffs, "basis": pot.moment_coeffs}
    _, want = O.loss_and_grad(O.OracleTables.from_potential(pot), params, (it, r, js, jt, cfg, 1, vols), targets)
    put = lambda a: torch.as_tensor(a, device="cuda")
    batch = DeviceBatch(put(it), put(r), put(js), put(jt), put(counts), put(cfg), put(vols), 1)
    tt = tuple(put(t) for t in targets)
    with MTPEngine(potential_path(name), N, stride) as eng:
        p = {k: torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for k, v in params.items()}
        weighted_loss(*predict(p, eng, batch), tt).backward()
        eng.sync_status()
    for k in want:
        assert np.abs(p[k].grad.cpu().numpy() - want[k]).max() <= 1e-8 * np.abs(want[k]).max(), k
