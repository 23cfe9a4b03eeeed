"""Plans whose shell pairs are more than kPlaceMaxPairs (6144, csrc/plan_build.cuh), which are ordered by
a radix sort and prefix sums, against plans of shorter lists, which are ordered by counting: a batch
against its molecules one by one, bit for bit, and the shards of a long list against the whole of it. (The
list of a shard plan is ordered by highest shell first, so that a quartet of one class can have bra and ket
the other way round: the two agree within the FP64 bar, 1e-12 each, and in which entries are zero.)"""
import numpy as np
import pytest

import molints_b200 as mi

pytestmark = pytest.mark.gpu


def _engine():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from molints_b200 import engine
    return torch, engine, engine.Engine(0)


def _run(torch, plan):
    out = torch.full((plan.npacked,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    plan.execute(out.data_ptr())
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("screen", [0.0, 1e-9])
@pytest.mark.parametrize("output", [1, 2])  # direct, two-phase
def test_batch_of_many_pairs(screen, output):
    torch, engine, eng = _engine()
    b = mi.basis
    mols = [b.synthetic_molecule(70 + m, h, n - h, *(b.POLARISED_C, b.POLARISED_H) if m == 1 else
                                 (b.SPLIT_VALENCE_HEAVY, b.SPLIT_VALENCE_H), 0.1, 5e3, f"m{m}")
            for m, (h, n) in enumerate([(5, 16), (2, 6), (6, 17), (5, 15), (6, 18), (4, 14), (5, 17), (1, 3)])]
    pairs = [m.nshell * (m.nshell + 1) // 2 for m in mols]
    assert sum(pairs) > 6144 > max(pairs)
    try:
        eng.set_stream(torch.cuda.current_stream().cuda_stream)
        kw = dict(screen_cutoff=screen, output=output)
        got = _run(torch, eng.plan_batch(mols, **kw)).cpu().numpy()
        at = 0
        for m in mols:
            one = _run(torch, eng.plan(m, **kw)).cpu().numpy()
            assert not np.isnan(one).any()
            assert np.array_equal(got[at:at + one.size], one), m.name
            at += one.size
        assert at == got.size
    finally:
        eng.set_stream(None)
        eng.close()


def test_shards_of_many_pairs():
    torch, engine, eng = _engine()
    rng = np.random.default_rng(17)
    rs = mi.basis._random_shell
    sh = mi.Shells.from_list([(rng.uniform(-8.0, 8.0, 3), int(s % 18 == 0), rs(rng, int(s % 18 == 0), 1 + s % 3, 0.3, 60.0))
                              for s in range(112)], "long")
    assert sh.nshell * (sh.nshell + 1) // 2 > 6144 and sh.npacked < 1 << 25
    try:
        eng.set_stream(torch.cuda.current_stream().cuda_stream)
        whole = _run(torch, eng.plan(sh)).cpu().numpy()
        parts = [_run(torch, eng.plan_shard(sh, r, 3)).cpu().numpy() for r in range(3)]
    finally:
        eng.set_stream(None)
        eng.close()
    assert not np.isnan(whole).any()
    parts = np.concatenate(parts)
    assert np.max(np.abs(parts - whole)) < 2e-12
    assert np.array_equal(parts == 0, whole == 0)
