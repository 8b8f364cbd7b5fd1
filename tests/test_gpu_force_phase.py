"""Basic moments, the force phase and the adjoint at the edges of their loads (GPU).

The kernel reads neighbours 16 bytes at a time, gives a lane one neighbour
(FP64) or two (FP32), and takes one of four chain layouts from the basis: the
level structure with offset 0, 1 or 2, or none.  Rows of 0 to 70 neighbours
and small bases of each layout, against the C++ FP64 oracle: 1e-10 relative in
FP64 (the drop-in bar); in mixed precision 1e-4 of the largest value (FP32
rounding, 6e-8, times about 1e3 terms of a sum, all of one sign at worst); the
coefficient gradient 1e-8 (its bar elsewhere) against torch double backward.
"""

import numpy as np
import pytest
import torch

from mtp_b200.engine import MTPEngine
from mtp_b200.mtp_file import MTPPotential, write_mtp
from mtp_b200.train import DeviceBatch, predict, weighted_loss
from oracle import mtp_oracle as O
from oracle.cpu_ref import CpuMTP

pytestmark = pytest.mark.gpu
COUNTS = [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 31, 32, 33, 40, 41, 42, 43, 63, 64, 65, 70, 0, 1]


def _potential(R, D, radial_functions, keep=lambda row: True):
    """Basic moments (mu, a, b, c) with mu < radial_functions(degree); a product m_k^2 for each."""
    basic = [(mu, a, b, c) for mu in range(R) for a in range(D + 1) for b in range(D + 1 - a)
             for c in range(D + 1 - a - b) if mu < radial_functions(a + b + c)]
    basic = [r for r in basic if keep(r)]
    B = len(basic)
    times = [(k, k, 1 + k % 3, B + k) for k in range(B)]
    rng = np.random.default_rng(R * 100 + D)
    mapping = [0] + list(range(B, 2 * B))
    return MTPPotential(
        scaling=1.0, species_count=2, min_dist=2.0, max_dist=5.0, radial_basis_type="RBChebyshev", radial_basis_size=6,
        radial_funcs_count=R, radial_coeffs=rng.normal(0, 0.1, (2, 2, R, 6)), alpha_moments_count=2 * B,
        alpha_index_basic_count=B, alpha_index_basic=np.array(basic), alpha_index_times_count=B,
        alpha_index_times=np.array(times), alpha_scalar_moments=B + 1, alpha_moment_mapping=np.array(mapping),
        species_coeffs=np.array([-1.0, -2.0]), moment_coeffs=rng.normal(0, 1.0, B + 1))


BASES = {
    "offset0_r1": lambda: _potential(1, 1, lambda v: 1),
    "offset0_r7": lambda: _potential(7, 12, lambda v: (12 - v) // 2 + 1),
    "offset1": lambda: _potential(6, 10, lambda v: min(6, (11 - v) // 2 + 1)),
    "offset2": lambda: _potential(6, 10, lambda v: min(6, (12 - v) // 2 + 1)),
    "no_structure": lambda: _potential(3, 5, lambda v: 3, keep=lambda r: (r[0] + r[1] + 2 * r[2] + r[3]) % 4 != 3),
    "no_structure_r8": lambda: _potential(8, 2, lambda v: 8),
}


def _rows(stride=72):
    rng = np.random.default_rng(11)
    N = len(COUNTS)
    r = rng.normal(size=(N, stride, 3))
    r *= (rng.uniform(2.0, 5.2, (N, stride)) / np.linalg.norm(r, axis=-1))[..., None]   # some past the cutoff
    js = rng.integers(0, N, (N, stride)).astype(np.int32)
    jt = rng.integers(0, 2, (N, stride)).astype(np.int32)
    it = rng.integers(0, 2, N).astype(np.int32)
    counts = np.array(COUNTS, dtype=np.int32)
    jt[np.arange(stride)[None] >= counts[:, None]] = -1
    return it, r, js, jt, counts


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("basis", sorted(BASES))
def test_rows_and_layouts_match_oracle(tmp_path, basis, precision):
    pot = BASES[basis]()
    path = str(tmp_path / "p.mtp")
    write_mtp(path, pot)
    it, r, js, jt, counts = _rows()
    N, stride = js.shape
    ref = CpuMTP(pot).compute(it, r, js, jt, counts)
    tol = 1e-10 if precision == "fp64" else 1e-4
    with MTPEngine(path, N, stride, precision=precision) as eng:
        for threads, apb in ((128, 1), (256, 2), (512, 4), (512, 1), (128, 4)):
            if precision == "fp64" and apb > 2:
                continue
            eng.set_launch(threads, 0, apb)
            out = eng.compute(it, r, js, jt, counts)
            for key in ("site_energies", "forces", "virial"):
                err = np.abs(out[key] - ref[key]).max() / np.abs(ref[key]).max()
                assert err <= tol, (threads, apb, key, err)


@pytest.mark.parametrize("basis,stride", [(b, 72) for b in sorted(BASES)] + [("offset2", 200)])
def test_adjoint_rows_and_layouts_match_oracle(tmp_path, basis, stride):
    pot = BASES[basis]()
    path = str(tmp_path / "p.mtp")
    write_mtp(path, pot)
    it, r, js, jt, counts = _rows(stride)
    N = len(it)
    cfg = np.sort(np.arange(N) % 3).astype(np.int32)
    js = np.where(cfg[np.clip(js, 0, N - 1)] == cfg[:, None], js, -1).astype(np.int32)
    vols = np.array([800.0, 900.0, 1000.0])
    rng = np.random.default_rng(3)
    targets = (rng.normal(size=3) * 10, rng.normal(size=(N, 3)), rng.normal(size=(3, 6)) * 1e-2)
    params = {"species": pot.species_coeffs, "radial": pot.radial_coeffs, "basis": pot.moment_coeffs}
    _, want = O.loss_and_grad(O.OracleTables.from_potential(pot), params, (it, r, js, jt, cfg, 3, vols), targets)
    dev = torch.device("cuda")
    put = lambda a: torch.as_tensor(a, device=dev)
    batch = DeviceBatch(put(it), put(r), put(js), put(jt), put(counts), put(cfg), put(vols), 3)
    tt = tuple(put(t) for t in targets)
    with MTPEngine(path, N, stride) as eng:
        for threads in (128, 256, 512):
            eng.set_launch(threads, 0, 0)
            p = {k: torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=True) for k, v in params.items()}
            weighted_loss(*predict(p, eng, batch), tt).backward()
            eng.sync_status()
            for k in ("species", "radial", "basis"):
                err = np.abs(p[k].grad.cpu().numpy() - want[k]).max() / np.abs(want[k]).max()
                assert err <= 1e-8, (threads, k, err)
