"""The bounded waits of the persistent cycle, made to run out by a CTA that holds back what
the others wait for: its arrival at the first cycle's counter, or that cycle's slots of the
nodes it shares.  The wait ends after about a second with OR_E_TIMEOUT and the number of a
CTA, whatever the waiting CTAs read in place of the slots, and the GPU stays usable.
"""
import numpy as np
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.OR_PREC_SPLIT, abi.OR_PREC_FP64], ids=["split", "fp64"])
@pytest.mark.parametrize("kind", ["shells", "hexas"])
@pytest.mark.parametrize("hook", ["OR_ECYCLE_TEST_STALL_CTA", "OR_ECYCLE_TEST_STALL_SLOTS"])
def test_wait_runs_out(monkeypatch, hook, kind, precision):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openradioss_b200 import build
    build.build()
    from openradioss_b200.ecycle import ECycle, ECycleError
    d = decks.c2_shell_plate(n=40, size=0.04) if kind == "shells" else decks.c1_hex_block(nx=8, ny=8, nz=32)
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    for cta in (1, 5):
        monkeypatch.setenv(hook, str(cta))
        g = ECycle(d, precision=precision)
        monkeypatch.delenv(hook)
        with pytest.raises(ECycleError) as ei:
            g.step(8)
        code, idx = g.error_info()
        assert ei.value.code == code == abi.OR_E_TIMEOUT
        assert 0 <= idx < nsm
        assert g.launch_count() == 1            # the persistent form
        torch.cuda.synchronize()                # the kernel returned; the context is usable
        g.close()
    h, r = ECycle(d, precision=precision), ECycle(d, precision=precision, persistent=-1)
    h.step(8)
    r.step(8)
    a, b = h.get_nodes()["d"], r.get_nodes()["d"]
    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
