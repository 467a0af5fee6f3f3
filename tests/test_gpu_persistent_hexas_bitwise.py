"""FP64 hexas in the persistent cycle against the patch and node kernels, bit for bit on the
build without contraction: the same operations in the same order, whatever way the forces take
between CTAs."""
import numpy as np
import pytest

from openradioss_b200 import abi, decks

pytestmark = pytest.mark.gpu


def block(nx, ny, nz, law, jcvt, extra_node=False):
    x, conn = decks.hex_block(nx, ny, nz, 1e-3)
    rng = np.random.Generator(np.random.PCG64(nx + 10 * ny + 100 * nz))
    base = np.isclose(x[:, 2], 0.0)
    x[~base] += rng.uniform(-5e-5, 5e-5, size=(int((~base).sum()), 3))
    if extra_node:                        # a node that no element touches moves on freely
        x = np.vstack([x, [0.1, 0.1, 0.1]])
        base = np.append(base, False)
    p = decks.new_part(x)
    decks.add_hex(p, conn, decks.steel_elastic() if law == 1 else decks.steel_jc(), decks.solid_prop(jcvt=jcvt))
    p["icodt"][base] = 7
    p["v"][~base] = [1.0, -0.5, -20.0]
    return decks.deck([p])


# one patch, a last patch of one hexa, exact patches, several CTAs; two and more patches a CTA
@pytest.mark.parametrize("n,law,jcvt,extra", [((3, 3, 3), 1, 0, False), ((5, 13, 1), 2, 0, True), ((4, 4, 4), 2, 1, False),
                                              ((11, 7, 19), 2, 1, True), ((20, 25, 30), 2, 0, False),
                                              ((23, 29, 31), 2, 1, True), ((28, 22, 47), 1, 0, False)])
def test_fp64_hexas_bitwise(n, law, jcvt, extra):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openradioss_b200 import build
    from openradioss_b200.ecycle import ECycle, load_library
    build.build()
    build.build(variant="nofma")
    lib = load_library(build.OUT_NOFMA)
    d = block(*n, law, jcvt, extra)
    p, r = (ECycle(d, precision=abi.OR_PREC_FP64, lib=lib, persistent=m) for m in (0, -1))
    for k in (1, 7, 32, 60):              # odd and even calls
        p.step(k)
        r.step(k)
        assert p.launch_count() == 1 and r.launch_count() > 1
        a, b = p.get_nodes(), r.get_nodes()
        for q in ("x", "d", "v"):
            assert np.array_equal(a[q], b[q]), (k, q)
        sa, sb = p.hex_state(0), r.hex_state(0)
        for q in sa:
            assert np.array_equal(sa[q], sb[q]), (k, q)
        assert p.time() == r.time()
    if law == 2 and max(n) > 5:
        assert sa["pla"].max() > 0
