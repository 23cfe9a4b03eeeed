"""Two-phase output against direct output, bit for bit, where the gather's column list and zero rows
have their edges: molecules of one function, of 44 to 46 functions (990, 1035 and 1081 columns around
the 1024-column steps of the list's index), with every pair zero but the diagonal ones, with no zero
pair at all, and of f shells (100-row pairs); alone, in one batch, FP64 and with quartet screening."""
import numpy as np
import pytest

import molints_b200 as mi

pytestmark = pytest.mark.gpu


def _mol(kind, n, seed):
    rng = np.random.default_rng(seed)
    rs = mi.basis._random_shell
    if kind == "one":
        return mi.Shells.from_list([((0.1, 0.2, 0.3), 0, [(1.1, 1.0)])])
    if kind == "far":  # tight s and p shells on centres 30 bohr apart: cross pairs vanish
        return mi.Shells.from_list([((30.0 * a, 0.0, 0.0), a % 2, rs(rng, a % 2, 1, 50.0, 90.0)) for a in range(n)])
    if kind == "f":
        return mi.Shells.from_list([(rng.uniform(-1.5, 1.5, 3), 3, rs(rng, 3, 1, 0.3, 2.0)) for _ in range(n // 10)])
    lst, left = [], n  # diffuse shells close together, n functions
    while left:
        l = min(int(rng.integers(0, 3)), 0 if left < 3 else 1 if left < 6 else 2)
        lst.append((rng.uniform(-2.0, 2.0, 3), l, rs(rng, l, int(rng.integers(1, 3)), 0.2, 3.0)))
        left -= mi.basis.ncart(l)
    return mi.Shells.from_list(lst)


MOLS = [("one", 1), ("near", 44), ("near", 45), ("near", 46), ("far", 24), ("f", 30)]


@pytest.mark.parametrize("screen", [0.0, 1e-9])
@pytest.mark.parametrize("pick", [[k] for k in range(len(MOLS))] + [list(range(len(MOLS)))])
def test_two_phase_edges(pick, screen):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from molints_b200 import engine
    mols = [_mol(*MOLS[k], seed=900 + k) for k in pick]
    eng = engine.Engine(0)
    outs = []
    try:
        eng.set_stream(torch.cuda.current_stream().cuda_stream)
        for output in (engine.OUTPUT_DIRECT, engine.OUTPUT_TWO_PHASE):
            plan = eng.plan_batch(mols, boys=engine.BOYS_EXACT, screen_cutoff=screen, output=output)
            out = torch.full((plan.npacked + 1,), float("nan"), dtype=torch.float64, device="cuda")
            for start in (0, 1):  # 16-byte aligned and not
                v = out[start:start + plan.npacked]
                v.fill_(float("nan"))
                plan.execute(v.data_ptr())
                torch.cuda.synchronize()
                outs.append(v.cpu().numpy().copy())
            plan.close()
    finally:
        eng.set_stream(None)
        eng.close()
    assert not np.isnan(outs[0]).any()
    for o in outs[1:]:
        assert np.array_equal(outs[0], o)
