"""Kernels that start before their predecessor in the stream has ended (csrc/launch.cuh).

What such a kernel reads may still be written while it is resident. Loads that want memory nobody writes
for the whole kernel (__ldg, or plain loads that __restrict__ turns into them) are therefore not used in one;
this is checked in the sources. On the GPU a chain that alternates between two buffers, as torch's allocator
hands them out, gives the results of the same calls waited for one by one, bit for bit."""
import ctypes as C
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "multem_b200" / "csrc"


def _sources():
    return {f.name: re.sub(r"//[^\n]*", "", f.read_text()) for f in sorted(CSRC.glob("*.cu*"))}


def _early_kernels():
    """(file, name, parameters, body) of every kernel whose body waits for its predecessor itself."""
    found = []
    for name, src in _sources().items():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(([^)]*)\)\s*\{", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            if "previous_done()" in src[m.end():i]:
                found.append((name, m.group(1), m.group(2), src[m.end():i]))
    return found


def test_kernels_that_start_early_use_ordinary_loads():
    early = _early_kernels()
    names = {k for _, k, _, _ in early}
    assert {"rows_kernel", "rows_pipe_kernel", "cols_kernel", "cols_pipe_kernel", "splat_kernel", "det_reduce_kernel",
            "ew_accumulate_kernel", "conv_kernel", "wgrad_kernel", "wgrad_finalize_kernel", "adam_kernel"} <= names
    for file, kernel, params, _ in early:
        assert "__restrict__" not in params, f"{file}: {kernel} has __restrict__ parameters"
    for file, src in _sources().items():
        if file in {f for f, _, _, _ in early} | {"fft_core.cuh", "mbarrier.cuh"}:
            assert not re.search(r"__ldg|ld\.global\.nc|const\s+\w+\*\s*__restrict__\s+\w+\s*=", src), f"{file}: non-coherent load"


def test_successors_start_after_the_wait():
    """No kernel lets its successor start before it has waited for its predecessor: two are resident, never three."""
    for file, kernel, _, body in _early_kernels():
        if "next_may_start()" in body:
            assert body.index("previous_done()") < body.index("next_may_start()"), f"{file}: {kernel}"


def test_tensor_memory_loads_wait_in_the_same_statement():
    """Registers of a tensor-memory load are undefined until its wait, and only one asm statement keeps their use behind it."""
    loads = 0
    for file, src in _sources().items():
        for m in re.finditer(r"asm\b[^;]*?\((?:[^()\"]|\"[^\"]*\"|\((?:[^()]|\([^()]*\))*\))*\)\s*;", src):
            if "tcgen05.ld" in m.group(0):
                loads += 1
                assert "tcgen05.wait::ld" in m.group(0), file
    assert loads >= 1


@pytest.mark.gpu
@pytest.mark.parametrize("B,ch,H,W", [(1, 16, 16, 16), (2, 40, 33, 17), (8, 32, 64, 64), (4, 256, 8, 8)])
def test_chain_over_alternating_buffers_equals_waited_calls(B, ch, H, W):
    torch = pytest.importorskip("torch")
    from multem_b200 import capi
    lib = capi.load()
    p = lambda t: C.c_void_p(t.data_ptr())
    g = torch.Generator().manual_seed(ch)
    w = [(torch.randn(ch, ch, 3, 3, generator=g) * (0.5 / ch) ** 0.5).to(torch.bfloat16).cuda() for _ in range(3)]
    b = [torch.randn(ch, generator=g).cuda() * 0.1 for _ in range(3)]
    x0 = torch.randn(B, ch, H, W, generator=g).to(torch.bfloat16).cuda()

    def chain(wait):
        buf = [x0.clone(), torch.zeros_like(x0)]
        dw, db = torch.zeros(ch, ch, 3, 3, device="cuda"), torch.zeros(ch, device="cuda")
        master, m, v = [torch.zeros(ch * ch * 9, device="cuda") for _ in range(3)]
        master.copy_(w[0].float().reshape(-1))
        wb = w[0].clone()
        torch.cuda.synchronize()
        calls = []
        for k in range(12):
            src, dst = buf[k % 2], buf[1 - k % 2]
            wk = wb if k % 3 == 0 else w[k % 3]
            calls += [lambda s=src, d=dst, q=wk, k=k: lib.mt_sg_conv3x3_forward(p(s), p(q), p(b[k % 3]), p(d), None, B, ch, ch, H, W, 1, None),
                      lambda s=src, d=dst: lib.mt_sg_add(p(s), p(d), p(s), s.numel(), None),
                      lambda s=src, d=dst: lib.mt_sg_conv3x3_backward_weight(p(s), p(d), p(d), p(dw), p(db), B, ch, ch, H, W, None),
                      lambda k=k: lib.mt_sg_adam(p(master), p(wb), p(dw), p(m), p(v), ch * ch * 9, 1e-4, 0.9, 0.999, 1e-8, k + 1, None),
                      lambda s=src, d=dst, q=wk: lib.mt_sg_conv3x3_backward_data(p(s), p(s), p(q), p(d), B, ch, ch, H, W, None)]
        for call in calls:
            capi.check(call())
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return buf + [dw, db, master, wb]

    ref = chain(True)
    assert all(t.isfinite().all() for t in ref)
    for _ in range(5):
        for got, want in zip(chain(False), ref):
            assert torch.equal(got, want)
