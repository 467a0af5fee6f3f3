"""The autotuner on one part of hexas, which runs a persistent cycle of its own."""
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.OR_PREC_SPLIT, abi.OR_PREC_FP64], ids=["split", "fp64"])
def test_hexa_block_times_both_forms(tmp_path, monkeypatch, precision):
    import json
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openradioss_b200 import autotune, build
    from openradioss_b200.ecycle import ECycle
    build.build()
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "cache.json"))
    d = decks.c1_hex_block(nx=10, ny=10, nz=40)
    key = autotune._key(d, precision, torch.cuda.get_device_name(0))
    # an entry that held the persistent cycle's time under the per-phase kernels' name
    old = {"block_hex": 64, "block_shell": 256, "persistent": -1, "ms_per_cycle": {"64": 1e-9}}
    json.dump({key: old}, open(autotune.CACHE, "w"))
    bh, bs, pers, ms = autotune.tune(d, precision, ncycles=64)
    assert set(ms) == {"64p", "64", "128", "256"}, ms      # tile 64 in both forms
    best = min(ms, key=ms.get)
    assert (bh, pers) == (int(best.rstrip("p")), 0 if best.endswith("p") else -1)
    h = ECycle(d, precision=precision, block_hex=bh, block_shell=bs, persistent=pers)
    h.step(64)
    assert (h.launch_count() == 1) == best.endswith("p")   # the form that was timed
    assert autotune.tune(d, precision, ncycles=64) == (bh, bs, pers, ms)     # from the cache
