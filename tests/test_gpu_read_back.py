"""get_nodes into pinned arrays, which a kernel fills directly up to 65,536 nodes for one array
and 262,144 for several, against pageable ones, which are always staged and copied: the same
bits, and nothing written beside them."""
import ctypes as C

import numpy as np
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu

GUARD = -7.25e300
KINDS = ("x", "d", "v", "vr")


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openradioss_b200 import build
    build.build()
    return torch


def strip(n):
    """n nodes: a strip of shells over the first ones, the others free and moving."""
    k = max(2, min(40, n // 2))
    x = np.zeros((max(n, 4), 3))
    i = np.arange(2 * k)
    x[:2 * k, 0], x[:2 * k, 1] = (i // 2) * 1e-3, (i % 2) * 1e-3
    x[2 * k:, 2] = 1e-2 + 1e-6 * np.arange(x.shape[0] - 2 * k)
    j = 2 * np.arange(k - 1)
    p = decks.new_part(x)
    decks.add_shell(p, np.stack([j, j + 2, j + 3, j + 1], 1), decks.steel_jc(), decks.shell_prop(1e-3))
    rng = np.random.Generator(np.random.PCG64(n))
    p["v"][:] = rng.uniform(-5, 5, x.shape)
    p["vr"][:2 * k] = rng.uniform(-5, 5, (2 * k, 3))
    return p


def free_node():
    """A part of one node that no element touches."""
    p = decks.new_part(np.array([[0.5, 0.25, -0.125]]))
    p["v"][:] = [1.0, 2.0, 3.0]
    return p


def call(h, part, arrays):
    dp = C.POINTER(C.c_double)
    h._call("get_nodes", part, *[None if a is None else C.cast(a.data_ptr(), dp) for a in arrays])


def check(torch, h, rows, kinds, pageable=()):
    """All parts' arrays of `kinds` in one allocation each, a guard row before every part and
    behind the last."""
    first = np.cumsum([1] + [r + 1 for r in rows])
    out = {}
    for pinned in (True, False):
        bufs = {}
        for k in kinds:
            t = torch.full((int(first[-1]), 3), GUARD, dtype=torch.float64)
            bufs[k] = t.pin_memory() if pinned and k not in pageable else t
        for p, r in enumerate(rows):
            call(h, p, [bufs[k][first[p]:first[p] + r] if k in bufs else None for k in KINDS])
        out[pinned] = bufs
    for k in kinds:
        a, b = out[True][k].numpy(), out[False][k].numpy()
        assert np.array_equal(a, b), k
        guards = np.concatenate([[0], first[1:] - 1])
        assert (a[guards] == GUARD).all(), k
        rest = np.delete(a, guards, axis=0)
        assert (rest != GUARD).all(), k


@pytest.mark.parametrize("precision", [abi.OR_PREC_SPLIT, abi.OR_PREC_FP64], ids=["split", "fp64"])
def test_parts_in_one_pinned_tensor(torch, precision):
    from openradioss_b200.ecycle import ECycle
    rows = [1, 127, 128, 129, 4, 1000]
    parts = [free_node() if r == 1 else strip(r) for r in rows]
    h = ECycle(decks.deck(parts), precision=precision)
    h.step(3)
    for kinds in (KINDS, ("x",), ("vr",), ("d", "v"), ("x", "vr")):
        check(torch, h, rows, kinds)
    check(torch, h, rows, KINDS, pageable=("v",))            # one array pageable: all staged
    h.close()


@pytest.mark.parametrize("precision", [abi.OR_PREC_SPLIT, abi.OR_PREC_FP64], ids=["split", "fp64"])
@pytest.mark.parametrize("n", [(1 << 16), (1 << 16) + 1, (1 << 18), (1 << 18) + 1])
def test_at_the_limits(torch, n, precision):
    from openradioss_b200.ecycle import ECycle
    h = ECycle(decks.deck([strip(n)]), precision=precision)
    h.step(2)
    for kinds in (("d",), ("d", "v"), KINDS):
        check(torch, h, [n], kinds)
    h.close()


def test_hexas_without_rotations(torch):
    """A model without rotational nodes: their velocities read zero, pinned or not."""
    from openradioss_b200.ecycle import ECycle
    d = decks.c1_hex_block(nx=3, ny=4, nz=5)
    h = ECycle(d)
    h.step(3)
    check(torch, h, [d["parts"][0]["x"].shape[0]], KINDS)
    t = torch.full((d["parts"][0]["x"].shape[0], 3), GUARD, dtype=torch.float64).pin_memory()
    call(h, 0, [None, None, None, t])
    assert (t.numpy() == 0).all()
    h.close()
