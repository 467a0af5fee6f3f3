"""Shells that share no nodes: a patch then holds four nodes per element, the most it can,
and needs the most shared memory, at the largest tile above all."""
import numpy as np
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu


def scattered(n, npt):
    """n quads of 1 mm, each with nodes of its own, one node of each held."""
    rng = np.random.Generator(np.random.PCG64(n))
    quad = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]], float) * 1e-3
    x = (quad[None] + 3e-3 * np.stack([np.arange(n) % 32, np.arange(n) // 32, 0 * np.arange(n)], 1)[:, None, :])
    x = (x + rng.uniform(-5e-5, 5e-5, x.shape)).reshape(-1, 3)
    p = decks.new_part(x)
    decks.add_shell(p, np.arange(4 * n).reshape(n, 4), decks.steel_jc(), decks.shell_prop(1e-3, npt=npt))
    p["v"][:] = rng.uniform(-5.0, 5.0, x.shape)
    p["icodt"][::4] = 7
    return decks.deck([p])


@pytest.mark.parametrize("precision", [abi.OR_PREC_SPLIT, abi.OR_PREC_FP64], ids=["split", "fp64"])
@pytest.mark.parametrize("tile", [64, 128, 256])
@pytest.mark.parametrize("n,npt", [(600, 5), (257, 3)])
def test_scattered_shells_at_every_tile(n, npt, tile, precision):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openradioss_b200 import build
    build.build()
    from openradioss_b200.ecycle import ECycle
    from oracle.oracle import Oracle
    d = scattered(n, npt)
    o = Oracle(d, nthreads=4)
    o.step(20)
    for form in (0, -1):
        h = ECycle(d, precision=precision, block_shell=tile, persistent=form)
        h.step(20)
        a, b = h.get_nodes()["d"], o.get_nodes()["d"]
        assert np.abs(a - b).max() <= (1e-10 if precision == abi.OR_PREC_FP64 else 1e-5) * np.abs(b).max()
        h.close()
