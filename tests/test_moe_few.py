"""The routed experts' products for a handful of pairs (csrc/moe.cu, ops.moe_few): an expert's pairs together or each for itself."""
import pytest
import torch


def test_where_the_pairs_of_an_expert_share_its_weights():
    from hos_b200 import ops
    together = lambda *a: ops.moe_few_plan(*a)[1] == ops.MOE_FEW_ROWS
    # (outputs, numbers each, pairs, experts[, gated]), with what a block per pair and per expert measured beside the rule
    for case in ((2304, 2048, 16, 16), (2304, 2048, 32, 16), (2304, 2048, 8, 16, True), (4096, 1024, 32, 16), (2048, 5632, 32, 4),
                 (14336, 2048, 32, 8), (8192, 4096, 2, 1, True)):
        assert together(*case), case
    for case in ((2304, 2048, 4, 16), (512, 1024, 32, 8, True), (512, 2048, 32, 8), (512, 16384, 32, 8), (256, 25000, 32, 4), (1024, 512, 4, 8),
                 (512, 30000, 8, 4), (1536, 3072, 4, 8), (2048, 14336, 32, 8)):
        assert not together(*case), case
    for features in (8, 64, 520, 2304, 30000):
        for k in (8, 512, 6144, 12288, 24576, 49152):
            for pairs in (1, 2, 7, 32):
                for experts in (1, 4, 128):
                    for gated in (False, True):
                        qf, rows = ops.moe_few_plan(features, k, pairs, experts, gated)
                        assert qf in (1, 2, 4) and rows in (1, ops.MOE_FEW_ROWS) and (rows == 1 or (4 * k <= 48 * 1024 and qf <= (2 if gated else 4)))


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("d,f", [(2048, 520), (8192, 264), (264, 8192), (12288, 64), (64, 12288), (25000, 40), (40, 25000)])
def test_a_pair_alone_and_in_company(d, f, gated):
    """Seven pairs on one expert (more than a block takes at a time), pairs with none beside them, a padding pair; rows of which a
    block holds four, three, two and one.  The bits are those of a pair by itself, whatever the features to a warp."""
    from hos_b200 import ops
    experts, top = 3, 2
    choice = [0, 1, 0, 2, 0, 1, -1, 0, 0, 2, 0, 1, 0, 1]
    n = len(choice) // top
    torch.manual_seed(d + f)
    h = torch.randn(n, d, device="cuda").bfloat16()
    ways = 2 if gated else 1
    w_up = (torch.randn(experts, ways * f, d, device="cuda") * d ** -0.5).bfloat16()
    w_down = (torch.randn(experts, d, f, device="cuda") * f ** -0.5).bfloat16()
    ids = torch.tensor(choice, dtype=torch.int32, device="cuda")
    weight = torch.rand(len(choice), device="cuda") + 0.5
    act = ops.EXPERT_ACTIVATIONS["gated_swish" if gated else "relu_square"]
    limit, alpha, shift = 7.0, 1.0, 0.0

    def run(ids, plan):
        y = torch.full((len(choice), f), 3.0, device="cuda").bfloat16()
        out = torch.full((len(choice), d), 3.0, device="cuda")
        assert ops.moe_few(h, w_up, w_down, ids, weight, y, out, top, experts, limit, alpha, shift, False, act, plans=(plan, plan))
        return y, out
    first = None
    for qf in (1, 2, 4):
        for rows in (1, ops.MOE_FEW_ROWS):
            y, out = run(ids, (qf, rows))
            assert bool((y[6] == 3.0).all()) and bool((out[6] == 3.0).all())       # nothing is written for a padding pair
            first = first or (y, out)
            assert torch.equal(y, first[0]) and torch.equal(out, first[1])
    for p in (0, 7, 12):
        lone = torch.full_like(ids, -1)
        lone[p] = choice[p]
        y, out = run(lone, (4, ops.MOE_FEW_ROWS))
        assert torch.equal(y[p], first[0][p]) and torch.equal(out[p], first[1][p])
    for p, e in enumerate(choice):
        if e < 0:
            continue
        x = w_up[e].double() @ h[p // top].double()
        if gated:
            g, u = x[:f].clamp(max=limit), x[f:].clamp(-limit, limit)
            want = g * torch.sigmoid(alpha * g) * (u + shift)
        else:
            want = x.clamp(min=0) ** 2
        err = (first[0][p].double() - want).norm() / want.norm()
        assert err < 4e-3, (p, float(err))                       # one rounding to 8 bits, half of 2^-8 at most
        want = weight[p].double() * (w_down[e].double() @ first[0][p].double())
        err = (first[1][p].double() - want).norm() / want.norm()
        assert err < 1e-5, (p, float(err))                       # 32-bit sums
