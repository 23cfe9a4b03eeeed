"""The generic kernel's units: quartets of several output tiles ((gg|gg): 50,625 outputs in tiles of
4096), contractions of more items (primitive quartet, root) than are set up at once (96), and
quartets of a few outputs, against the long-double HGP restatement.  Tolerance as for the other g
bases: the FP64 bar 1e-12 plus twice the FP64 restatement's own error on the basis."""
import numpy as np
import pytest

import molints_b200 as mi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shells", [
    ((4, 4),),              # one centre, (gg|gg): 13 tiles, 256 primitive quartets x 9 roots
    ((4, 1), (3, 2)),       # tiles of exactly and just over 4096 outputs do not occur: (gg|gf) 33,750
    ((0, 7), (4, 2)),       # (gs|ss): 15 outputs, 686 primitive quartets x 3 roots
    ((1, 3), (2, 2), (4, 1)),
])
def test_units_against_oracle(oracle, shells):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from molints_b200 import engine
    rng = np.random.default_rng(4 * len(shells) + sum(k for _, k in shells))
    lst = [(xyz, l, mi.basis._random_shell(rng, l, k, 0.3, 8.0))
           for xyz in ((0.0, 0.1, -0.2), (0.7, -0.9, 0.4))[:1 if len(shells) == 1 else 2] for l, k in shells]
    sh = mi.Shells.from_list(lst, "units")
    eng = engine.Engine(0)
    try:
        got = eng.eri_packed(sh, boys=engine.BOYS_EXACT)
    finally:
        eng.close()
    with oracle.exact_boys(), oracle.stable_orientation():
        ld = oracle.eri_packed_hgp_ld(sh, nthreads=0)
        floor = 2.0 * float(np.max(np.abs(oracle.eri_packed_hgp(sh, nthreads=0) - ld)))
    err = float(np.max(np.abs(got - ld)))
    print(f"{shells}: {got.size} integrals, |GPU - ld| {err:.2e}, floor {floor:.2e}")
    assert err < 1e-12 + floor
