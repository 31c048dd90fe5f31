"""Plans that run in two lanes of L2-sized chunks by default (from their
second exec on): every exec gives the same bits, in order, captured in a
CUDA graph, and without the second lane."""
import numpy as np
import pytest

from oracle import oracle as O
from sip_b200 import _lib as L

pytestmark = pytest.mark.gpu

# chunk counts with a remainder; 3-D items, 3-D slabs, small 2-D items, a 2-D item per chunk
CASES = [([65536], 131, 0), ([40000], 420, 0), ([64, 64, 64], 41, 0), ([98, 128, 147], 4, 0), ([256, 256, 200], 1, 0),
         ([256, 256], 131, 0), ([2000, 2000], 3, 0), ([65536], 131, 1)]


@pytest.mark.parametrize("sizes,batch,pulse", CASES)
def test_chunked_execs_agree(cuda, monkeypatch, sizes, batch, pulse):
    from sip_b200.fft import FftHandle, check

    torch = cuda
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(sizes) + batch)
    x = torch.randn((batch, *sizes), generator=g, device="cuda", dtype=torch.complex64)
    filt = torch.randn(sizes[-1], generator=g, device="cuda", dtype=torch.complex64)

    def plan():
        h = FftHandle()
        check(h.set_hint(L.SIP_FFT_HINT_RUNTIME_COMPILE, 1), "hint")
        if pulse:
            rc = h.make_plan_pulse_1d(sizes[0], batch, filt.data_ptr(), 0)
        else:
            make = {1: h.make_plan_1d, 2: h.make_plan_2d, 3: h.make_plan_3d}[len(sizes)]
            rc = make(*sizes, L.ASCEND_FFT_C2C, L.ASCEND_FFT_FORWARD, batch)
        check(rc, "plan")
        h.bind_workspace()
        return h

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    monkeypatch.setenv("SIP_FFT_L2_CHUNK_MB", "0")
    whole = plan()
    check(whole.set_stream(s), "stream")
    want = torch.empty_like(x)
    check(whole.exec_c2c(x, want), "whole")
    monkeypatch.delenv("SIP_FFT_L2_CHUNK_MB")
    h = plan()
    check(h.set_stream(s), "stream")
    assert any(gr["chunk_units"] < gr["units"] for gr in h.describe()["chunk_groups"])
    for _ in range(3):  # the first exec runs whole passes, the others two lanes
        y = torch.zeros_like(x)
        s.wait_stream(torch.cuda.current_stream())
        check(h.exec_c2c(x, y), "exec")
        s.synchronize()
        assert torch.equal(torch.view_as_real(y), torch.view_as_real(want))
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        check(h.exec_c2c(x, y), "captured")
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(torch.view_as_real(y), torch.view_as_real(want))
    if not pulse:
        rows = min(batch, 2)
        ref = torch.fft.fftn(x[:rows].to(torch.complex128), dim=tuple(range(1, x.dim()))).cpu().numpy()
        assert O.rel_l2(y[:rows].cpu().numpy(), ref) <= 1e-6
    del graph
    h.destroy()
    whole.destroy()
