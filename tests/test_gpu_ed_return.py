"""A sector Lanczos call without a vector leaves nothing of its own on the stream: H = 0 breaks down in the first
iteration, with the second one already enqueued."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_nothing_left_running():
    torch = pytest.importorskip("torch")
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import abi, nqs
    nqs.set_options()
    perm, chars = nqs._perm_args(*nqs.kagome_perm(2, 3, "translations", "A1"))
    e, r = C.c_double(), abi.LanczosResult()
    run = nqs.lib().nqs_lanczos_e0_kagome_heisenberg_projected_lean
    args = (2, 3, 0.0, 1, nqs._ip(perm), nqs._dp(chars), len(chars), 50, 1e-9, C.byref(e), C.byref(r))
    assert run(*args) == 0
    query = torch.cuda.ExternalStream(nqs.lib().nqs_gpu_stream()).query
    for _ in range(20):
        assert run(*args) == 0
        assert query()
    assert r.iterations == 1 and e.value == 0.0
