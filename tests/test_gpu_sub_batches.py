"""How a small batched multiply is cut: whole by default, and into the sub-batches the
caller asks for once it has chosen their number or least size; the products are the
same. What a call takes of the scratch arena shows the cut: two sub-batches of three
pairs have two regions of two pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _context():
    import kunpbfv_b200 as kb
    return kb.BFVContext.from_bits(12, [36, 36], [37], 65537, dnum=2)


@pytest.mark.parametrize("choose", ["set_branches", "branches", "min_branch_pairs"])
def test_the_callers_choice_holds_for_small_batches(choose):
    import kunpbfv_b200 as kb
    from kunpbfv_b200 import tune
    ctx = _context()
    sch = kb.BFVScheme(ctx, b"\x61" * 32)
    sch.addMultKey_23(kb.SecretKey(ctx, b"\x62" * 32))
    a, b = (kb.Ciphertext(ctx, tune._random_pairs(ctx, 3, s)) for s in (1, 2))
    out = kb.Ciphertext(ctx, count=3)
    plan = sch.mult_relin_plan(a, b, out)
    plan.launch()
    want = sch.mult_relin(a, b).cipher_device
    assert torch.equal(out.cipher_device, want)
    one = ctx.scratch_bytes(1)
    low = ctx.at_level(1)
    low_one = low.scratch_bytes(1)
    assert ctx.scratch_bytes(3) == 3 * one and low.scratch_bytes(3) == 3 * low_one, "whole by default"
    if choose == "set_branches":
        ctx.set_branches(2)
    else:
        ctx.tune_set(choose, ctx.tune_get(choose))
        assert low.scratch_bytes(3) == 4 * low_one, "levels follow the knobs"
    assert ctx.scratch_bytes(3) == 4 * one, "two sub-batches"
    assert torch.equal(sch.mult_relin(a, b).cipher_device, want)
    out.cipher_device.zero_()
    plan.launch()
    assert torch.equal(out.cipher_device, want) and plan.info() == (2, 2), "the plan follows"
    ctx.tune_set("min_branch_pairs", 2)
    assert ctx.scratch_bytes(3) == 3 * one, "no sub-batch of two pairs in three"
