"""Captured executes in the orders in which programs call them: a graph launched again, another output,
two outputs in turn, back to the first, and after the context's scratch has moved, for direct plans,
two-phase plans (gather and zero rows on their own streams) and screened ones; every execute writes the
whole output, bit for bit what an uncaptured one writes."""
import pytest

import molints_b200 as mi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("output,screen", [(1, 0.0), (1, 1e-9), (2, 0.0), (2, 1e-9)])
def test_sequences(output, screen):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from molints_b200 import engine
    b = mi.basis
    mols = [b.synthetic_molecule(40 + m, 2, 5, b.POLARISED_C, b.POLARISED_H, 0.1, 1e4, f"g{m}") for m in range(2)]
    big = [b.synthetic_molecule(50 + m, 3, 8, b.SPLIT_VALENCE_HEAVY, b.SPLIT_VALENCE_H, 0.1, 5e3, f"b{m}")
           for m in range(5)]
    eng = engine.Engine(0)
    try:
        eng.set_stream(torch.cuda.current_stream().cuda_stream)
        plan = eng.plan_batch(mols, screen_cutoff=screen, output=output)
        ref = torch.full((plan.npacked,), float("nan"), dtype=torch.float64, device="cuda")
        plan.execute(ref.data_ptr())
        torch.cuda.synchronize()
        assert not torch.isnan(ref).any()
        plan.set_graph(True)
        outs = [torch.empty_like(ref) for _ in range(2)]

        def sequence(order):
            for k in order:
                outs[k].fill_(float("nan"))
                plan.execute(outs[k].data_ptr())
                torch.cuda.synchronize()
                assert torch.equal(outs[k], ref), (order, k)

        sequence([0, 0, 0, 1, 1, 1, 0])
        sequence([0, 0, 1, 0, 1, 0, 1, 1])
        # a larger two-phase plan: the scratch is allocated anew
        other = eng.plan_batch(big, output=engine.OUTPUT_TWO_PHASE)
        o2 = torch.empty(other.npacked, dtype=torch.float64, device="cuda")
        other.execute(o2.data_ptr())
        sequence([1, 1, 1, 0, 0, 0])
        plan.set_graph(False)
        sequence([0, 1])
        plan.set_graph(True)
        sequence([1, 1, 1])
        other.close()
        plan.close()
    finally:
        eng.set_stream(None)
        eng.close()
