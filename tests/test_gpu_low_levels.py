"""The lowest levels (GPU): levels 2 and 4 have scalar moments only (monomials of
degree 0), level 2 no products either.  Against the C++ FP64 oracle (1e-10
relative; mixed: FP32 rounding, 6e-8, times about 1e3 terms) and, for the
coefficient gradient, torch double backward (1e-8)."""

import numpy as np
import pytest
import torch

from mtp_b200 import basis as B
from mtp_b200.engine import MTPEngine
from mtp_b200.mtp_file import with_random_coeffs, write_mtp
from mtp_b200.train import DeviceBatch, predict, weighted_loss
from oracle import mtp_oracle as O
from oracle.cpu_ref import CpuMTP

pytestmark = pytest.mark.gpu


def _case(tmp_path, level, n=11, stride=37):
    pot = with_random_coeffs(B.template_potential(level, 2, min_dist=2.0, max_dist=5.0), seed=level)
    path = str(tmp_path / "p.mtp")
    write_mtp(path, pot)
    rng = np.random.default_rng(level)
    r = rng.normal(size=(n, stride, 3))
    r *= (rng.uniform(2.1, 5.2, (n, stride)) / np.linalg.norm(r, axis=-1))[..., None]
    counts = np.resize([stride, 0, 1, 2, stride - 1], n).astype(np.int32)
    jt = rng.integers(0, 2, (n, stride)).astype(np.int32)
    jt[np.arange(stride)[None] >= counts[:, None]] = -1
    return pot, path, (rng.integers(0, 2, n).astype(np.int32), r, rng.integers(0, n, (n, stride)).astype(np.int32), jt,
                       counts)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("level", [2, 4, 6, 8])
def test_low_levels_match_oracle(tmp_path, level, precision):
    pot, path, rows = _case(tmp_path, level)
    ref = CpuMTP(pot).compute(*rows)
    tol = 1e-10 if precision == "fp64" else 1e-4
    with MTPEngine(path, len(rows[0]), rows[1].shape[1], precision=precision) as eng:
        for threads, apb in ((0, 0), (128, 1), (128, 2), (512, 2), (512, 1), (256, 4)):
            if precision == "fp64" and apb > 2:
                continue
            if threads:
                eng.set_launch(threads, 0, apb)
            out = eng.compute(*rows)
            for key in ("site_energies", "forces", "virial"):
                assert np.abs(out[key] - ref[key]).max() <= tol * np.abs(ref[key]).max(), (threads, apb, key)


@pytest.mark.parametrize("level", [2, 4, 6])
def test_adjoint_of_low_levels(tmp_path, level):
    pot, path, (it, r, js, jt, counts) = _case(tmp_path, level)
    N = len(it)
    cfg, vols = np.zeros(N, dtype=np.int32), np.array([700.0])
    rng = np.random.default_rng(3)
    targets = (rng.normal(size=1) * 10, rng.normal(size=(N, 3)), rng.normal(size=(1, 6)) * 1e-2)
    params = {"species": pot.species_coeffs, "radial": pot.radial_coeffs, "basis": pot.moment_coeffs}
    _, want = O.loss_and_grad(O.OracleTables.from_potential(pot), params, (it, r, js, jt, cfg, 1, vols), targets)
    put = lambda a: torch.as_tensor(a, device="cuda")
    batch = DeviceBatch(put(it), put(r), put(js), put(jt), put(counts), put(cfg), put(vols), 1)
    tt = tuple(put(t) for t in targets)
    with MTPEngine(path, N, r.shape[1]) as eng:
        p = {k: torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for k, v in params.items()}
        weighted_loss(*predict(p, eng, batch), tt).backward()
        eng.sync_status()
    for k in want:
        assert np.abs(p[k].grad.cpu().numpy() - want[k]).max() <= 1e-8 * np.abs(want[k]).max(), k
