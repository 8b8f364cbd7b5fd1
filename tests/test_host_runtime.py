"""Host code of the library on a CUDA runtime without a GPU.

The library's objects are linked with tests/host/fake_cudart.cpp: device memory
is host memory, kernels do not run, and the runtime calls are logged.  What is
checked here is what the host does: which allocations, copies and launches it
makes, in which order, and what it refuses while a stream is being captured."""

import ctypes
import os
import re
import subprocess

import pytest

from conftest import REPO, potential_path
from mtp_b200._lib import EFLAG, REUSE_NEIGHBORS, SIGNATURES, VFLAG

CSRC = os.path.join(REPO, "jax-mtp_b200", "csrc")
FP64, MIXED = 0, 1
L16, L20, L24, L28 = "cfg1_L16_S2.mtp", "cfg3_L20_S2.mtp", "cfg2_L24_S3.mtp", "cfg4_L28_S4.mtp"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    subprocess.run(["make", "-C", CSRC, "-j", "4"], check=True, capture_output=True)
    out = str(tmp_path_factory.mktemp("host") / "libmtp_host.so")
    objs = [os.path.join(CSRC, "_build", f"mtp_{n}.o") for n in ("model", "kernels", "train", "md", "abi")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include",
                    os.path.join(REPO, "tests", "host", "fake_cudart.cpp"), *objs, "-o", out], check=True)
    L = ctypes.CDLL(out)
    for name, (res, args) in SIGNATURES.items():
        getattr(L, name).restype, getattr(L, name).argtypes = res, args
    L.fake_log.restype, L.fake_stream.restype = ctypes.c_char_p, ctypes.c_void_p
    L.fake_capture.argtypes = [ctypes.c_void_p, ctypes.c_int]
    L.fake_set_device.argtypes = [ctypes.c_void_p, ctypes.c_int]
    L.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
    return L


class Handle:
    """One handle with device buffers for its capacities, on a stream of the caller."""

    def __init__(self, lib, name, atoms, stride, precision=FP64):
        self.L, self.stride, self.h = lib, stride, ctypes.c_void_p()
        assert lib.mtp_create(potential_path(name).encode(), atoms, stride, 5.0, 0, precision,
                              ctypes.byref(self.h)) == 0
        self.stream = lib.fake_stream()
        lib.mtp_set_stream(self.h, self.stream)
        sizes = dict(itypes=4 * atoms, rijs=24 * atoms * stride, js=4 * atoms * stride, jtypes=4 * atoms * stride,
                     counts=4 * atoms, forces=24 * atoms, energy=8, virial=48)
        self.buf = {k: self.alloc(n) for k, n in sizes.items()}
        lib.fake_clear()

    def alloc(self, n):
        p = ctypes.c_void_p()
        assert self.L.cudaMalloc(ctypes.byref(p), n) == 0
        return p.value

    def compute(self, n, flags=EFLAG | VFLAG, stride=None, energy=None, virial=None):
        """Status and log of one device call."""
        b = self.buf
        self.L.fake_clear()
        st = self.L.mtp_compute_device(self.h, n, stride or self.stride, b["itypes"], b["rijs"], b["js"], b["jtypes"],
                                       b["counts"], flags, energy or b["energy"], b["forces"],
                                       virial or b["virial"], None, None)
        return st, self.log()

    def adjoint(self, n):
        b = self.buf
        if "cfg" not in b:
            b.update(cfg=self.alloc(4 * n), volumes=self.alloc(8), gE=self.alloc(8), gF=self.alloc(24 * n),
                     gS=self.alloc(48), gspecies=self.alloc(1 << 16), gmoment=self.alloc(1 << 16),
                     gradial=self.alloc(1 << 16))
        return self.L.mtp_adjoint_batch_device(self.h, n, self.stride, 1, b["itypes"], b["rijs"], b["js"],
                                               b["jtypes"], b["counts"], b["cfg"], b["volumes"], b["gE"], b["gF"],
                                               b["gS"], b["gspecies"], b["gmoment"], b["gradial"])

    def noalloc(self, n):
        b = self.buf
        self.L.fake_clear()
        st = self.L.mtp_compute_device_noalloc(self.h, n, self.stride, b["itypes"], b["rijs"], b["js"], b["jtypes"],
                                               b["counts"], b["energy"], b["forces"], b["virial"])
        return st, self.log()

    def captured(self, n, **kw):
        """The same call while its stream is captured."""
        self.L.fake_capture(self.stream, 1)
        try:
            return self.compute(n, **kw)
        finally:
            self.L.fake_capture(self.stream, 0)

    def log(self):
        return self.L.fake_log().decode()

    def set_launch(self, threads, atoms):
        assert self.L.mtp_set_launch(self.h, threads, 0, atoms) == 0

    def launch(self):
        out = (ctypes.c_int * 5)()
        assert self.L.mtp_get_launch(self.h, out) == 0
        return dict(zip(("threads", "blocks", "smem", "per_sm", "atoms"), out))

    def error(self):
        return self.L.mtp_last_error(self.h).decode()

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.L.mtp_destroy(self.h)


@pytest.mark.parametrize("precision,stride", [(FP64, 12), (MIXED, 600)])
def test_global_value_space_never_moves(lib, precision, stride):
    """A captured graph keeps the address of the value space in global memory:
    no later call of the handle may free it, whatever its number of atoms."""
    with Handle(lib, L28, 700, stride, precision) as h:
        assert h.compute(100)[0] == 0
        for n in (400, 256, 149, 700, 297, 1):
            st, log = h.compute(n)
            assert st == 0
            assert "free" not in log, f"{n} atoms"


def test_global_value_space_is_there_for_a_captured_size(lib):
    """A size whose value spaces are more than those of the calls before it."""
    with Handle(lib, L28, 4000, 12) as h:
        assert h.compute(200)[0] == 0 and h.launch()["atoms"] == 2
        st, log = h.captured(4000)
        assert st == 0 and "in-capture" not in log, h.error()


@pytest.mark.parametrize("first,second,atoms", [(4000, 100, 2), (100, 4000, 1)])
def test_capture_in_global_memory_uses_the_programs_that_are_there(lib, first, second, atoms):
    with Handle(lib, L28, 4000, 12) as h:
        assert h.compute(first)[0] == 0
        st, log = h.captured(second)
        assert st == 0 and "in-capture" not in log, h.error()
        assert h.launch()["atoms"] == atoms
        assert h.compute(second)[0] == 0 and h.launch()["atoms"] == 3 - atoms


def test_capture_in_shared_memory_uses_the_programs_that_are_there(lib):
    with Handle(lib, L24, 20000, 12, MIXED) as h:
        assert h.compute(20000)[0] == 0
        ran = h.launch()
        st, log = h.captured(100)
        assert st == 0 and "in-capture" not in log, h.error()
        assert (h.launch()["threads"], h.launch()["atoms"]) == (ran["threads"], ran["atoms"])


def test_allocation_free_call_after_a_training_gradient(lib):
    """The gradient's programs (ordered for 16-byte operands) serve rows that are
    too long for four atoms per block, the width's own shape."""
    with Handle(lib, L20, 100, 400, MIXED) as h:
        assert h.noalloc(100)[0] != 0            # nothing uploaded
        assert h.adjoint(100) == 0
        st, log = h.noalloc(100)
        assert st == 0, h.error()
        assert "malloc" not in log and "k_mtp_eval" in log


def test_coefficients_wait_for_work_on_the_stream_before(lib):
    """An evaluation on the legacy default stream may still read the old values
    when the handle has moved to its own, non-blocking stream."""
    with Handle(lib, L16, 100, 12) as h:
        lib.mtp_set_stream(h.h, None)
        assert h.compute(100)[0] == 0
        lib.mtp_use_own_stream(h.h)
        lib.fake_clear()
        species = (ctypes.c_double * 2)(1.0, 2.0)
        assert lib.mtp_set_coeffs(h.h, species, None, None) == 0
        lines = h.log().splitlines()
        copy = next(x for x in lines if x.startswith("memcpy"))
        assert copy.endswith("stream (nil)") and lines[-1] == "synchronize stream (nil)", lines


def test_coefficients_refused_in_a_capture(lib):
    with Handle(lib, L16, 100, 12) as h:
        species = (ctypes.c_double * 2)(1.0, 2.0)
        lib.fake_capture(h.stream, 1)
        lib.fake_clear()
        st = lib.mtp_set_coeffs(h.h, species, None, None)
        lib.fake_capture(h.stream, 0)
        assert st != 0 and "memcpy" not in h.log()


def _totals(log):
    return re.search(r"totals energy (\S+) virial (\S+)", log).groups()


def test_totals_of_another_device_are_copied(lib):
    """Peer memory may not be mapped on this device: kernels do not store there."""
    with Handle(lib, L16, 100, 12) as h:
        e, v = h.alloc(8), h.alloc(48)
        lib.fake_set_device(e, 1)
        st, log = h.compute(100, energy=e, virial=v)
        assert st == 0 and _totals(log) == ("(nil)", hex(v))
        assert re.search(rf"memcpy-async {hex(e)} 8 ", log)


def test_totals_at_odd_addresses_are_copied(lib):
    with Handle(lib, L16, 100, 12) as h:
        e, v = h.alloc(16) + 4, h.alloc(56) + 4
        st, log = h.compute(100, energy=e, virial=v)
        assert st == 0 and _totals(log) == ("(nil)", "(nil)")
        assert re.search(rf"memcpy-async {hex(e)} 8 ", log) and re.search(rf"memcpy-async {hex(v)} 48 ", log)


def test_lists_of_a_call_that_failed_are_sorted_by_the_next(lib):
    """The incoming lists are sorted by the force gather: a call that fails
    between the two leaves that to the call that reuses them."""
    with Handle(lib, L16, 2000, 12) as h:
        lib.fake_fail_malloc(1)                  # the upload of the programs, after the lists
        st, log = h.compute(2000)
        assert st != 0 and "k_fill_incoming" in log and "k_force_gather" not in log
        st, log = h.compute(2000, flags=EFLAG | VFLAG | REUSE_NEIGHBORS)
        assert st == 0 and "k_fill_incoming" not in log and "k_force_gatherILb1E" in log
        st, log = h.compute(2000, flags=EFLAG | VFLAG | REUSE_NEIGHBORS)
        assert st == 0 and "k_force_gatherILb0E" in log


SIZES = (1, 100, 149, 593, 1185, 5000)


@pytest.mark.parametrize("name,precision,threads,atoms", [(L20, MIXED, 512, 4), (L20, MIXED, 512, 1), (L20, FP64, 256, 2),
                                                         (L24, MIXED, 512, 4), (L24, MIXED, 128, 2), (L16, MIXED, 128, 4),
                                                         (L28, FP64, 512, 2), (L28, FP64, 512, 1)])
def test_requested_shape_is_pinned(lib, name, precision, threads, atoms):
    with Handle(lib, name, max(SIZES), 12, precision) as h:
        h.set_launch(threads, atoms)
        for n in SIZES:
            assert h.compute(n)[0] == 0
            assert (h.launch()["threads"], h.launch()["atoms"]) == (threads, atoms), n


@pytest.mark.parametrize("name,precision", [(L16, FP64), (L20, MIXED), (L24, MIXED), (L28, FP64)])
def test_requested_threads_fix_the_shape_for_every_size(lib, name, precision):
    with Handle(lib, name, max(SIZES), 12, precision) as h:
        for threads in (128, 256, 512):
            h.set_launch(threads, 0)
            shapes = set()
            for n in SIZES:
                assert h.compute(n)[0] == 0
                shapes.add((h.launch()["threads"], h.launch()["atoms"]))
            assert len(shapes) == 1
            if name != L28:                      # in global memory: always 512 threads
                assert shapes.pop()[0] == threads


def test_requested_threads_that_do_not_fit_give_way_to_fewer(lib):
    with Handle(lib, L28, 1000, 450, MIXED) as h:   # 512 threads fit up to 448 slots, 256 up to 452
        h.set_launch(512, 1)
        for n in (1, 1000):
            assert h.compute(n)[0] == 0
            assert (h.launch()["threads"], h.launch()["atoms"]) == (256, 1)


# Rows that each shape took, and blocks per SM, with neighbour-major staging rows:
# (potential, precision, threads, atoms per block, slots, blocks per SM)
ROWS = [(L16, MIXED, 128, 4, 80, 4), (L16, MIXED, 128, 4, 116, 3), (L16, MIXED, 256, 4, 183, 2), (L16, MIXED, 128, 2, 184, 4),
        (L16, FP64, 128, 2, 80, 4), (L16, FP64, 256, 2, 170, 2), (L20, MIXED, 256, 4, 88, 2), (L20, MIXED, 128, 4, 40, 3),
        (L20, FP64, 256, 2, 100, 2), (L20, FP64, 128, 2, 45, 3), (L24, MIXED, 512, 4, 72, 1), (L24, MIXED, 256, 4, 77, 1),
        (L24, MIXED, 128, 4, 80, 1), (L24, MIXED, 256, 2, 74, 2), (L24, MIXED, 128, 2, 77, 2), (L24, FP64, 512, 2, 76, 1),
        (L24, FP64, 256, 2, 82, 1), (L24, FP64, 128, 2, 85, 1), (L28, MIXED, 512, 1, 409, 1)]


@pytest.mark.parametrize("name,precision,threads,atoms,slots,per_sm", ROWS)
def test_row_lengths_that_fit(lib, name, precision, threads, atoms, slots, per_sm):
    with Handle(lib, name, 2, slots, precision) as h:
        h.set_launch(threads, atoms)
        assert h.compute(2)[0] == 0
        got = h.launch()
        assert (got["threads"], got["atoms"]) == (threads, atoms) and got["per_sm"] >= per_sm


def test_failed_upload_of_the_tables_is_made_up_for(lib):
    """Whichever allocation of the first call fails, the next call has all of them."""
    live = lambda log: log.count("malloc 0x") - log.count("free 0x")
    with Handle(lib, L16, 100, 12) as h:
        whole = live(h.compute(100)[1])
    for n in range(1, whole + 1):
        with Handle(lib, L16, 100, 12) as h:
            lib.fake_fail_malloc(n)
            st, log = h.compute(100)
            assert st != 0 and "malloc-failed" in log
            left = live(log)
            st, log = h.compute(100)
            assert st == 0, h.error()
            assert left + live(log) == whole, n


@pytest.mark.parametrize("n", [100, 296, 600])
def test_mixed_rows_in_global_memory_take_one_atom_per_block(lib, n):
    """Two take 2.3 times as long as one (level 28, rows of 500 slots)."""
    with Handle(lib, L28, 600, 500, MIXED) as h:
        for threads, atoms in ((0, 0), (512, 2)):
            if threads:
                h.set_launch(threads, atoms)
            assert h.compute(n)[0] == 0 and h.launch()["atoms"] == 1
