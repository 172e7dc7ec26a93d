"""A wait that ran out is reported by the call it happened in and by no later one, before and after
the process has made an asynchronous call (the two ways the status word is cleared and read)."""
import numpy as np
import pytest

import blaze_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["native", "split"])
def test_timeout_is_reported_once(method):
    torch = pytest.importorskip("torch")
    n = 256
    A = torch.from_numpy(O.uniform(n * n, 1)).cuda().view(n, n)
    B = torch.from_numpy(O.uniform(n * n, 2)).cuda().view(n, n)
    C = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    ref = (A @ B).cpu().numpy()

    def call(**kw):
        G.dgemm_ex(O.ROW_MAJOR, O.NO_TRANS, O.NO_TRANS, n, n, n, 1.0, A, n, B, n, 0.0, C, n, G.opts(method=method, **kw))

    for asynchronous in (False, True):
        if asynchronous:
            call(synchronous=False, stream=torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
        G.lib().gb300_debug_inject_stall(1, 20_000_000)
        with pytest.raises(G.Gb300Error) as ei:
            call()
        assert ei.value.status == G.ERR_DEVICE_TIMEOUT
        for _ in range(2):
            call()
            assert np.allclose(C.cpu().numpy(), ref, rtol=1e-12, atol=1e-12)
        G.synchronize()
