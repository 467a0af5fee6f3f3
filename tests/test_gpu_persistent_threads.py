"""Handles of several host threads, each in its own stream, whose persistent cycles compete for
the SMs: every handle gives the bits it gives alone."""
import threading

import numpy as np
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu


def run(d, precision, calls):
    from openradioss_b200.ecycle import ECycle
    h = ECycle(d, precision=precision)
    for n in calls:
        h.step(n)
    assert h.launch_count() == 1
    out = h.get_nodes()
    h.close()
    return out


def test_concurrent_handles():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openradioss_b200 import build
    build.build()
    jobs = [(decks.c1_hex_block(nx=20, ny=20, nz=45, law=decks.LAW_JOHNSON_COOK), abi.OR_PREC_FP64),
            (decks.c1_hex_block(nx=33, ny=35, nz=40), abi.OR_PREC_SPLIT),
            (decks.c1_hex_block(nx=5, ny=5, nz=20), abi.OR_PREC_SPLIT),
            (decks.c2_shell_plate(n=150, size=0.15), abi.OR_PREC_SPLIT)]
    calls = [40] * 60 + [1, 7] * 20
    alone = [run(d, p, calls) for d, p in jobs]
    got, errors = [None] * len(jobs), []

    def work(i):
        try:
            got[i] = run(*jobs[i], calls)
        except Exception as e:            # reported by the test, not by the thread
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(alone, got):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
