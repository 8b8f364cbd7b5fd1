"""Energy and virial totals after launches that overlapped on the same scratch (GPU).

Overlapping allocation-free calls share one scratch array and may spoil each
other's totals; the calls after them must not be affected.  The overlapping
calls here have no atoms, so that the totals kernel (whose blocks count
themselves in the shared array) is all that they run beside each other."""

import numpy as np
import pytest
import torch

from conftest import golden_case, potential_path
from mtp_b200.engine import MTPEngine

pytestmark = pytest.mark.gpu


def test_calls_after_an_overlap():
    g = golden_case("bcc54_L16")
    path = potential_path(str(g["potential"]))
    N, n = g["js"].shape
    dev = torch.device("cuda")
    rows = [torch.as_tensor(np.ascontiguousarray(g[k]).astype(t), device=dev)
            for k, t in (("itypes", np.int32), ("rijs", np.float64), ("js", np.int32), ("jtypes", np.int32),
                         ("counts", np.int32))]
    none = [r[:0] for r in rows]
    out = lambda m: (torch.zeros(1, dtype=torch.float64, device=dev),
                     torch.zeros((m, 3), dtype=torch.float64, device=dev),
                     torch.zeros(6, dtype=torch.float64, device=dev))
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    with MTPEngine(path, N, n) as a, MTPEngine(path, N, n) as b:
        want = [t.clone() for t in a.compute_device(*rows)]
        b.compute_device(*rows)
        o0, o1, o2 = out(N), out(0), out(0)
        torch.cuda.synchronize()
        for _ in range(200):
            a.compute_device_noalloc(*none, *o1, stream=s1)
            b.compute_device_noalloc(*none, *o2, stream=s2)
        torch.cuda.synchronize()
        for _ in range(2):
            a.compute_device_noalloc(*rows, *o0)
            torch.cuda.synchronize()
            a.sync_status()
            for x, y in zip(o0, want):
                assert (x - y).abs().max() <= 1e-10 * y.abs().max()
