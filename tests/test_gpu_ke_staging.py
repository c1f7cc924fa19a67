"""The element stiffness of the drop-in kernels reaches the host through a buffer that a thread keeps: it is
usable whatever modes were on when it was made."""
import threading

import pytest
import torch

from genpipeline_gb300 import cuda_kernels

pytestmark = pytest.mark.gpu


def _call():
    x, p = torch.ones(1, device="cuda"), torch.arange(24.0, device="cuda")
    edof = torch.arange(24, device="cuda").reshape(1, 24)
    return cuda_kernels.fused_spmv(x, p, torch.eye(24, device="cuda"), edof, 3.0, 1, 1, 1).cpu()


def _in_thread(fn):
    got = []

    def run():
        try:
            fn()
        except BaseException as e:  # a thread's exception is lost otherwise
            got.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    if got:
        raise got[0]


def test_made_in_inference_mode():
    def run():
        with torch.inference_mode():
            _call()
        assert torch.equal(_call(), torch.arange(24.0))

    _in_thread(run)


def test_made_with_a_default_device():
    def run():
        with torch.device("cuda"):
            y = _call()
        assert torch.equal(y, torch.arange(24.0))

    _in_thread(run)
