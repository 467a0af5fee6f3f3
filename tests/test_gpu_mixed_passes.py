"""The two element passes of a mixed mesh, run side by side, against the same passes in turn.

With programmatic launches (OR_ECYCLE_PDL, read when a handle is created) the hexa kernel
starts beside the shell kernel and takes the node pass's results through a flag that the
shells release; without them every kernel waits for the one before.  The arithmetic is the
same, so nodes, element state, energies and time are equal bit for bit.
"""
import numpy as np
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu


def final(d, n, **kw):
    from openradioss_b200.ecycle import ECycle
    h = ECycle(d, **kw)
    for k in (n, 33, 1):                   # graph replays and single cycles, from either parity
        h.step(k)
    parts = range(len(d["parts"]))
    hexes = sum(len(p["hex"]) for p in d["parts"])
    shells = sum(len(p["shell"]) for p in d["parts"])
    out = {f"{p}.{k}": v for p in parts for k, v in h.get_nodes(p).items()}
    out.update({f"hex{g}.{k}": v for g in range(hexes) for k, v in h.hex_state(g).items()})
    out.update({f"shell{g}.{k}": v for g in range(shells) for k, v in h.shell_state(g).items()})
    scalars = [(h.energies(p), h.time(p)) for p in parts]
    h.close()
    return out, scalars


# the flat block's 360,000 hexas are several waves and its 7,200 shells fewer patches than
# SMs; the parts mix meshes of one kind; the small block is one wave of both; the staged
# shell kernel is forced on a mesh whose shells would not choose it
@pytest.mark.parametrize("precision", [abi.OR_PREC_SPLIT, abi.OR_PREC_FP64], ids=["split", "fp64"])
@pytest.mark.parametrize("deck,cycles,staged", [("flat", 320, None), ("parts", 96, None), ("small", 64, None),
                                                ("flat", 32, "1")])
def test_passes_side_by_side_bitwise(monkeypatch, deck, cycles, staged, precision):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openradioss_b200 import build
    build.build()
    if staged:
        monkeypatch.setenv("OR_ECYCLE_SHELL_STAGED", staged)
    d = {"flat": lambda: decks.c4_mixed_mesh(nx=200, ny=200, nz=9),
         "parts": lambda: decks.c3_batched_parts(nparts=10, scale=0.3),
         "small": lambda: decks.c4_mixed_mesh(nx=5, ny=13, nz=7)}[deck]()
    r = []
    for flag in ("1", "0"):
        monkeypatch.setenv("OR_ECYCLE_PDL", flag)
        r.append(final(d, cycles, precision=precision))
    (a, sa), (b, sb) = r
    assert sa == sb
    assert a.keys() == b.keys()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
