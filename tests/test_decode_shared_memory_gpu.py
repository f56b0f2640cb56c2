"""The decode attention's kernels keep the shared memory that they were given (csrc/attention_decode.cu), in whatever order groups of
other sizes ask for theirs."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# two query heads to a kv head take a ring of three stages, eight a ring of two: the same kernel, with more and with less shared memory
ORDER = """
import torch
from hos_b200 import ops
from hos_b200.parts import attention_fast as af
HD, N, L = 256, 24, 300
pos = torch.full((N,), L - 1, dtype=torch.int32, device="cuda")
row = torch.arange(N, dtype=torch.int32, device="cuda")
table = torch.arange(N * 5, dtype=torch.int32, device="cuda").view(N, 5)
torch.manual_seed(1)

def run(nh, nkv, splits):
    pages = [torch.randn(N * 5, nkv, 64, HD, device="cuda", generator=torch.Generator("cuda").manual_seed(i)).bfloat16() for i in (2, 3)]
    q = torch.randn(N, nh * HD, device="cuda", generator=torch.Generator("cuda").manual_seed(4)).bfloat16()
    out = torch.empty_like(q)
    af.decode(q, nh * HD, out, pos, row, row, ops.PagedKVArgs(*pages, table, 0, nkv, HD), N, nh, 0.06, 0.0, None, L, n_splits=splits, max_new=1)
    torch.cuda.synchronize()
    return out

first = run(8, 4, 2)                                        # 192 items: no clusters, a ring of three stages
assert af.clusters_fit(HD, 32, 4, 2) >= 0                   # eight heads to a kv head: asks about a smaller one
assert torch.equal(run(8, 4, 2), first)
run(32, 4, 2)
assert af.clusters_fit(HD, 8, 4, 2) >= 0
run(32, 4, 1)
assert torch.equal(run(8, 4, 2), first)
print("all ran")
"""


@pytest.mark.gpu
def test_groups_of_other_sizes_in_any_order():
    got = subprocess.run([sys.executable, "-c", ORDER], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert got.returncode == 0 and "all ran" in got.stdout, got.stderr[-2000:]
