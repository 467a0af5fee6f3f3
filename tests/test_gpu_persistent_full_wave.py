"""Persistent cycles whose CTAs have an element on every thread: six patches of 64 shells or of
64 FP64 hexas, twelve of split hexas (47,361 shells and more on 148 SMs).  No warp is left for
the time step, which the warp that hands in last then sends; in FP64 the shells' points do not
fit in shared memory any more."""
import numpy as np
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nofma():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openradioss_b200 import build
    from openradioss_b200.ecycle import load_library
    build.build()
    build.build(variant="nofma")
    return load_library(build.OUT_NOFMA)


def patches_a_cta(nel, tile):
    import torch
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    return -(-(-(-nel // tile)) // nsm)


@pytest.mark.parametrize("precision", [abi.OR_PREC_SPLIT, abi.OR_PREC_FP64], ids=["split", "fp64"])
@pytest.mark.parametrize("npt,tile,kw", [(5, 64, {}), (5, 128, {}), (3, 64, {}), (2, 64, {}), (5, 64, dict(ishell=3))])
def test_shells_on_every_thread(nofma, precision, npt, tile, kw):
    """Bit for bit the phase kernels' results, in plastic flow, over odd and even calls."""
    from openradioss_b200.ecycle import ECycle
    d = decks.c2_shell_plate(n=225, size=0.225, npt=npt, **kw)
    part = d["parts"][0]
    part["v"][part["icodt"] == 0, 2] = 35.0
    part["icodt"][part["icodt"] != 0] = 7
    assert patches_a_cta(225 * 225, tile) * tile == 384
    p, r = (ECycle(d, precision=precision, lib=nofma, persistent=m, block_shell=tile) for m in (0, -1))
    for n in (1, 24, 15):
        p.step(n)
        r.step(n)
    assert p.persistent_info()[0] and p.launch_count() == 1 and r.launch_count() > 1
    a, b = p.get_nodes(), r.get_nodes()
    for k in ("x", "d", "v", "vr"):
        assert np.array_equal(a[k], b[k]), k
    sa, sb = p.shell_state(0), r.shell_state(0)
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
    assert np.abs(sa["pla"]).max() > 0
    assert p.time() == r.time()


@pytest.mark.parametrize("precision,n,threads", [(abi.OR_PREC_FP64, (37, 37, 39), 64), (abi.OR_PREC_SPLIT, (45, 50, 48), 32)],
                         ids=["fp64", "split"])
def test_hexas_on_every_thread(nofma, precision, n, threads):
    from openradioss_b200.ecycle import ECycle
    d = decks.c1_hex_block(*n, law=decks.LAW_JOHNSON_COOK, vz=-20.0)
    assert patches_a_cta(n[0] * n[1] * n[2], 64) * threads == 384
    p, r = (ECycle(d, precision=precision, lib=nofma, persistent=m) for m in (0, -1))
    for k in (1, 24, 15):
        p.step(k)
        r.step(k)
    assert p.launch_count() == 1 and r.launch_count() > 1
    a, b = p.get_nodes()["d"], r.get_nodes()["d"]
    assert np.abs(a - b).max() <= (1e-10 if precision == abi.OR_PREC_FP64 else 1e-5) * np.abs(b).max()
    assert p.time()["ncycle"] == r.time()["ncycle"] == 40
