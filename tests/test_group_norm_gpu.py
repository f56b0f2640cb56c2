"""group_norm_gate (csrc/postnorm.cu) over wide groups: a block that holds its row."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("groups,size", [(1, 512), (1, 516), (1, 1024), (1, 1028), (1, 2048), (1, 2052), (1, 4100), (1, 8192), (1, 8196),
                                         (3, 2056), (1, 1001)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("per_group", [False, True])
def test_wide_groups(groups, size, dtype, per_group):
    """Around the widths at which a thread holds 1, 2, 4 and 8 pieces, and widths that are no whole pieces or too wide; a padding
    row; both activations.  Sums of `size` squares in 32-bit, a few roundings after it."""
    from hos_b200 import ops
    n, act = 5, ops.ACT_LOGISTIC if per_group else ops.ACT_X_LOGISTIC
    torch.manual_seed(size)
    o = torch.randn(n, groups * size, device=DEV)
    gate = torch.randn(n, 8 + groups * size, device=DEV) * 2
    w = torch.rand(size if per_group else groups * size, device=DEV) + 0.5
    seq = torch.tensor([0, 1, -1, 2, 3], dtype=torch.int32, device=DEV)
    out = torch.full((n, groups * size), 7.0, device=DEV, dtype=dtype)
    ops.group_norm_gate(o, w, gate, 8, act, seq, out, 1e-6, groups, size)
    x = o.double().view(n, groups, size)
    x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w.double().view(1, -1, size)
    z = gate[:, 8:].double().view(n, groups, size)
    want = (x * torch.sigmoid(z) * (1.0 if per_group else z)).flatten(1)
    want[2] = 0.0
    err = (out.double() - want).abs() / want.abs().clamp(min=1.0)
    assert err.max().item() <= (4e-6 if dtype == torch.float32 else 4e-3)
