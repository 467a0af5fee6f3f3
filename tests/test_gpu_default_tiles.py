"""The hexa tile that the library picks in the split form between 113,664 and 132,608 hexas
(148 SMs), told from the results: patch sums are added per patch, so their rounding names
the tile."""
import numpy as np
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu


def block(nx, ny, nz):
    return decks.c1_hex_block(nx, ny, nz, law=decks.LAW_JOHNSON_COOK)["parts"][0]


@pytest.mark.parametrize("parts,tile", [
    (lambda: [block(40, 50, 60)], 128),                                                # one part
    (lambda: [block(20, 50, 60), block(20, 25, 60), block(20, 25, 60)], 64),           # several, to 13 patches an SM
    (lambda: [block(20, 50, 62), block(20, 25, 62), block(20, 25, 62)], 128),          # beyond
    (lambda: [block(20, 50, 60), block(20, 50, 60)] + decks.c2_shell_plate(n=30, size=0.03)["parts"], 128),
], ids=["one", "several", "beyond", "with a plate"])
def test_split_hexas_past_the_persistent_reach(parts, tile):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes for 148 SMs")
    from openradioss_b200 import build
    from openradioss_b200.ecycle import ECycle
    build.build()
    d = decks.deck(parts())
    out = {}
    for t in (None, 64, 128):
        h = ECycle(d, precision=abi.OR_PREC_SPLIT, **({} if t is None else {"block_hex": t}))
        h.step(40)
        assert h.launch_count() > 1
        out[t] = h.get_nodes(0)["v"]
        h.close()
    assert not np.array_equal(out[64], out[128])
    assert np.array_equal(out[None], out[tile])
