"""The delta rule four tokens at a time (csrc/state_scan.cu) against 64 bits and beside the walk token by token."""
import ctypes
import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def case(dim, vdim, H, Gk, lens, fresh, seed=0, hard=False):
    """Rows as conv_prep leaves them (keys of length 1, queries scaled by dim^-1/2), columns before them, padding rows."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = sum(lens)
    rows = torch.randn(n + 3, 4 + 2 * Gk * dim + H * vdim, device=DEV, generator=g)
    qk = rows[:, 4:4 + 2 * Gk * dim].view(n + 3, 2 * Gk, dim)
    qk /= qk.norm(dim=-1, keepdim=True)
    if hard:                                         # neighbours' keys nearly alike: the inverse is as far from I as it gets
        qk[1:, Gk:] = qk[:1, Gk:] + 0.05 * qk[1:, Gk:]
        qk /= qk.norm(dim=-1, keepdim=True)
    qk[:, :Gk] *= dim ** -0.5
    decay = torch.exp(-torch.rand(n + 3, H, device=DEV, generator=g) * 0.2)
    decay[5::17] = 0.0                               # everything is forgotten, and nearly everything
    decay[11::23] = 1e-30
    beta = torch.ones(n + 3, H, device=DEV) if hard else torch.rand(n + 3, H, device=DEV, generator=g)
    if hard:
        decay.fill_(1.0)
    state = torch.randn(len(lens) + 2, H, vdim, dim, device=DEV, generator=g)
    cu = [0]
    for length in lens:
        cu.append(cu[-1] + length)
    pos = torch.cat([torch.arange(length) + (0 if f else 7) for length, f in zip(lens, fresh)] + [torch.zeros(3)]).int().to(DEV)
    seq = torch.cat([torch.full((length,), i) for i, length in enumerate(lens)] + [torch.full((3,), -1)]).int().to(DEV)
    slots = torch.arange(len(lens), 0, -1, dtype=torch.int32, device=DEV)
    step = SimpleNamespace(token_pos=pos, token_seq=seq, cu_seqlens=torch.tensor(cu, dtype=torch.int32, device=DEV), seq_slot=slots,
                           n_seqs=len(lens), n_tokens=n + 3, max_new=max(lens))
    return rows, decay, beta, state, step


def run(c, dim, vdim, H, Gk, fours, o_mult=1.0):
    from hos_b200 import ops
    rows, decay, beta, state, step = c
    state = state.clone()
    out = torch.full((rows.shape[0], H * vdim), 7.0, device=DEV)
    was, ops.fours_of_tokens = ops.fours_of_tokens, fours
    try:
        ops.state_scan(rows, 4, 4 + Gk * dim, 4 + 2 * Gk * dim, False, decay, True, beta, state, step, out, H, Gk, dim, vdim, o_mult=o_mult)
    finally:
        ops.fours_of_tokens = was
    return out, state


def exact(c, dim, vdim, H, Gk, o_mult=1.0):
    rows, decay, beta, state, step = c
    x, state = rows.double(), state.double().clone()
    q, k = (x[:, 4 + i * Gk * dim:4 + (i + 1) * Gk * dim].view(-1, Gk, dim).repeat_interleave(H // Gk, 1) for i in (0, 1))
    v = x[:, 4 + 2 * Gk * dim:].view(-1, H, vdim)
    out = torch.full((rows.shape[0], H, vdim), 7.0, dtype=torch.float64, device=DEV)
    cu = step.cu_seqlens.tolist()
    for i, slot in enumerate(step.seq_slot.tolist()):
        S = state[slot] if int(step.token_pos[cu[i]]) else torch.zeros_like(state[slot])
        for t in range(cu[i], cu[i + 1]):
            S = S * decay[t].double()[:, None, None]
            u = beta[t].double()[:, None] * (v[t] - torch.einsum("hvd,hd->hv", S, k[t]))
            S = S + u[:, :, None] * k[t][:, None]
            out[t] = o_mult * torch.einsum("hvd,hd->hv", S, q[t])
        state[slot] = S
    return out.flatten(1), state


@pytest.mark.parametrize("dim,vdim,H,Gk", [(64, 64, 4, 2), (128, 128, 4, 2), (128, 20, 3, 3), (256, 36, 2, 1), (64, 8, 2, 2)])
@pytest.mark.parametrize("lens,fresh", [((32,), (1,)), ((65, 94, 99), (0, 1, 0)), ((200, 1, 31, 130), (1, 0, 0, 1))])
@pytest.mark.parametrize("hard", [False, True])
def test_against_64_bits(dim, vdim, H, Gk, lens, fresh, hard):
    """Chunks and fours that are full, cut and of one token; sequences that start and go on; decays of zero, of 1e-30 and of one; keys nearly
    alike; value columns that do not fill a block.  A number of the read-outs is a sum of some hundred products of numbers up to
    about one, each rounded to 2^-24 of itself, and a state's cell carries on what its predecessors lost: 200 x 2^-24 x 10.  And
    the fours are not further off than the walk is (1.5 times its error at most, for the luck of few numbers)."""
    c = case(dim, vdim, H, Gk, lens, fresh, hard=hard)
    want, want_state = exact(c, dim, vdim, H, Gk, 0.5)
    n = sum(lens)
    errors = []
    for fours in (True, False):
        out, state = run(c, dim, vdim, H, Gk, fours, 0.5)
        assert bool((out[n:] == 7.0).all()) and torch.equal(state[0], c[3][0]) and torch.equal(state[-1], c[3][-1])
        err = [(out[:n].double() - want[:n]).abs().max().item(), (state.double() - want_state).abs().max().item()]
        assert max(err) <= 200 * 2.0 ** -24 * 10, (fours, err)
        errors.append([(out[:n].double() - want[:n]).norm().item(), (state.double() - want_state).norm().item()])
    assert all(a <= 1.5 * b + 1e-7 * math.sqrt(n) for a, b in zip(*errors)), errors


def test_which_calls_go_by_fours():
    from hos_b200 import ops
    f = ops.mixers().lib.hos_state_scan_fours
    f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_int] * 6
    assert f(31, 1, 16, 128, 128, 31) == 0 and f(32, 1, 16, 128, 128, 32) == (32 // 4 + 2) * 16 * 28
    assert f(100, 4, 16, 128, 128, 97) == 0                              # few tokens a sequence
    assert f(2048, 1, 16, 100, 128, 2048) == 0 and f(2048, 1, 16, 128, 130, 2048) == 0
