"""Which products of a plan leave partial tiles: only those whose output the operation recorded next adds up, whatever parts an
arrangement is put together from (the step walker fails a step whose operation does not take them)."""
import pytest
import torch

from gibbs_b200.engine import plan as P
from gibbs_b200.ops import hybrid
from gibbs_b200.parts.base import Runtime
from gibbs_b200.parts.block import SandwichResidual
from gibbs_b200.parts.norm import PlainRMSNorm
from gibbs_b200.parts.runner import BranchPart

D = 256


class Recorder(P.PlanBuilder):
    def keep(self, t):
        return 0 if t is None else t.data_ptr()


class Product(BranchPart):
    """A sublayer whose last product is its last operation."""

    def __init__(self):
        self.weight = torch.zeros(D, D, dtype=torch.bfloat16)

    def run(self, rn, h, out, caches=None):
        rn.branch_linear(h, self.weight, None, out)


class WorksOnItsOutput(Product):
    def run(self, rn, h, out, caches=None):
        super().run(rn, h, out, caches)
        rn.op("act_rows", [out.data_ptr(), out.stride(0), out.data_ptr(), 1, out.stride(0), rn.N, D, 0])


class ProductBehind(Product):
    """Reads its output through a second product."""

    def run(self, rn, h, out, caches=None):
        super().run(rn, h, out, caches)
        again = rn.buffer("again", D, torch.float32)
        rn.linear(out, self.weight.float(), None, again)
        rn.branch_linear(again, self.weight.float(), None, out)


class OwnAddition(PlainRMSNorm):
    """A norm behind a sublayer with an operation of its own."""

    def add_normed(self, rn, x, y, copy=None, then=None):
        rn.op("scaled_sum", [x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), self.gain.data_ptr(), 0, 0, 0, rn.N, D], [1.0])
        return super().add_normed(rn, x, y, copy, then)


class ReadsAfterwards(PlainRMSNorm):
    def add_normed(self, rn, x, y, copy=None, then=None):
        out = super().add_normed(rn, x, y, copy, then)
        rn.op("scaled_sum", [x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), self.gain.data_ptr(), 0, 0, 0, rn.N, D], [1.0])
        return out


@pytest.mark.parametrize("mixer,norm,tiles", [
    (Product, PlainRMSNorm, True), (WorksOnItsOutput, PlainRMSNorm, False), (ProductBehind, PlainRMSNorm, False), (Product, OwnAddition, False),
    (Product, ReadsAfterwards, False),
])
def test_tiles_are_left_only_to_an_operation_that_adds_them(mixer, norm, tiles):
    rt = Runtime(device=torch.device("cpu"), dtype=torch.bfloat16)
    make = lambda cls: cls({"dim": D, "eps": 1e-5}, {"weight": torch.ones(D)}, rt)
    block = SandwichResidual({"mixer_norm": make(PlainRMSNorm), "mixer": mixer(), "mixer_post_norm": make(norm), "ffn_norm": make(PlainRMSNorm),
                              "ffn": Product(), "ffn_post_norm": make(PlainRMSNorm)}, rt)
    plan = Recorder(rt, D, cap=512, max_requests=4, with_tensorcore=True)
    block.plan_ops(plan, [])
    assert len(plan.ops) >= 5
    left = []
    for record, behind in zip(plan.ops, plan.ops[1:] + [None]):
        if record["op"] == P.P_LINEAR and int(record["flags"]) & P.LF_PARTIALS:
            assert behind is not None and int(behind["op"]) == hybrid.plan_id("norm_add") and int(behind["flags"]) & hybrid.TAKES_PARTIALS
            left.append(record)
        elif behind is not None:
            assert not int(behind["flags"]) & hybrid.TAKES_PARTIALS
    assert len(left) == 1 + int(tiles)             # (the feed-forward's, and the mixer's where nothing comes between)
