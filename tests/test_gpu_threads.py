"""Engines and network layers on several host threads at once (the handles may be used from different threads):
launches of one kernel with shared memory of different sizes must not disturb each other."""
import ctypes as C
import threading

import numpy as np
import pytest

from multem_b200 import api, capi, specimens

pytestmark = pytest.mark.gpu


def _together(works, n):
    """Run every function of `works` n times on a thread of its own, starting together."""
    start, errors = threading.Barrier(len(works)), []

    def loop(f):
        start.wait()
        try:
            for _ in range(n):
                f()
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(f,)) for f in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def _wave_of(n_types):
    p = specimens.hrtem_si001(nx=64, ny=64, na=2, nb=2, nc=1)
    p.pn_nconf = 64
    atoms = p.spec_atoms.copy()
    atoms[:, 0] = [6 + i % n_types for i in range(len(atoms))]
    p.spec_atoms = atoms
    return p


def test_specimens_of_different_numbers_of_elements(monkeypatch):
    monkeypatch.setenv("MTB_GRAPH", "0")  # every run launches its kernels anew,
    monkeypatch.setenv("MTB_EW_BATCH", "1")  # the splat once per configuration
    works, engines = [], []
    for n_types in (1, 16, 3):
        e = api.Engine(_wave_of(n_types))
        ref = e.run()["data"]

        def work(e=e, ref=ref):
            for a, b in zip(e.run()["data"], ref, strict=True):
                np.testing.assert_array_equal(a["psi_coh"], b["psi_coh"])

        works.append(work)
        engines.append(e)
    _together(works, 100)
    for e in engines:
        e.close()


def test_convolutions_of_different_tiles():
    torch = pytest.importorskip("torch")
    lib = capi.load()
    p = lambda t: C.c_void_p(t.data_ptr())
    works = []
    # the same kernel (16 output channels, one pixel tile) with the least and with the most shared memory
    for B, Cin, Cout, H, W in ((1, 4, 8, 4, 8), (1, 40, 8, 2, 126), (1, 64, 16, 3, 140)):
        g = torch.Generator().manual_seed(Cin)
        x = torch.randn(B, Cin, H, W, generator=g).to(torch.bfloat16).cuda()
        w = torch.randn(Cout, Cin, 3, 3, generator=g).to(torch.bfloat16).cuda()
        y = torch.empty(B, Cout, H, W, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()

        def run(x=x, w=w, y=y, s=stream, d=(B, Cin, Cout, H, W)):
            capi.check(lib.mt_sg_conv3x3_forward(p(x), p(w), None, None, p(y), *d, 0, C.c_void_p(s.cuda_stream)))

        run()
        torch.cuda.synchronize()
        ref = torch.nn.functional.conv2d(x.double(), w.double(), padding=1)
        assert float((y - ref).norm() / ref.norm()) < 1e-5
        works.append(run)
    _together(works, 3000)
    torch.cuda.synchronize()
