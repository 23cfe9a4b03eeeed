"""The class kernels around the Boys switch (T = 30 in the reference mode, 40 in the exact one), where
near lanes read the tables and far lanes run the same recurrences with constants: s and p shells on two
centres whose distances sweep T across both switches, against the long-double HGP restatement in the
same mode.  The integrals are below 1 in magnitude and the kernels' errors a few 1e-16 of the largest
intermediate; 1e-13 also covers a value at the switch itself taken from the other branch (the two
differ by e^-T there, 1e-13 of F at T = 30 times F < 0.2)."""
import numpy as np
import pytest

import molints_b200 as mi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["reference", "exact"])
@pytest.mark.parametrize("t", [0.0, 1.0 / 64, 12.3, 29.999999999, 30.0, 30.000000001, 39.999999999, 40.0,
                               40.000000001, 41.7, 500.0])
def test_around_the_switch(oracle, mode, t):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from molints_b200 import engine
    # (aa|bb) of s shells with exponents 1.3 on A and 0.7 on B: zeta = 2.6, eta = 1.4, T = rho R^2
    rho = 2.6 * 1.4 / (2.6 + 1.4)
    r = np.sqrt(t / rho)
    lst = [(c, l, [(e, 1.0)]) for c, e in (((0.0, 0.0, 0.0), 1.3), ((0.0, r, 0.0), 0.7)) for l in (0, 1)]
    # a shell between the centres, so that chunks mix near and far quartets
    lst.append(((0.2, 0.5 * r, -0.1), 0, [(2.1, 0.4), (0.3, 0.6)]))
    sh = mi.Shells.from_list(lst, "switch")
    eng = engine.Engine(0)
    try:
        got = eng.eri_packed(sh, method=engine.METHOD_HGP,
                             boys=engine.BOYS_EXACT if mode == "exact" else engine.BOYS_REFERENCE)
    finally:
        eng.close()
    if mode == "exact":
        with oracle.exact_boys():
            ref = oracle.eri_packed_hgp_ld(sh, nthreads=4)
    else:
        ref = oracle.eri_packed_hgp_ld(sh, nthreads=4)
    assert np.max(np.abs(got - ref)) < 1e-13
