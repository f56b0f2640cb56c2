"""Attention over a compressed (latent) cache.

Per position the layer keeps ONE row shared by all heads: the latent c (`kv_rank` numbers: the
first rows of the down projection, RMS-normed with a weight) and one rotated key part (`rot_dim`
numbers, not normed).  A head's key is [W_uk_h c | rotated part], its value W_uv_h c, its query
[dim unrotated | rot_dim rotated] numbers; the score is their dot product times `scale`.  The
mask is causal with an optional window of the last `window` keys; with `sink`, a learned number
per head joins the softmax's denominator as exp(sink_h) (no key, no value, unscaled).

Prompts of many rows whose sizes fit form keys and values (one product of the latents, then the tcgen05 walk of
csrc/latent_prompt.cu: less arithmetic per pair).  Elsewhere neither is formed: the query absorbs W_uk (q'_h = W_uk_h^T q_h, `kv_rank`
numbers) and W_uv is applied to the weighted sum of latents, so the attention kernel reads
`kv_rank + rot_dim` numbers per key for all heads.  Everything between the projections (norm of
c, angles, scores, softmax, weighted sums) is 32-bit; with bfloat16 rows the two products run on the
tensor cores with every 32-bit operand as two bfloat16 terms (csrc/latent_attention.cu).

With `q_rank` the queries go through a latent of their own: one product makes [query latent | latent | key part] from
the layer's input, the query latent is RMS-normed with a weight, and a second product expands it into the heads' queries.

The rotation may pair neighbouring numbers or halves (the position part's style).

Cache: one keys-only group of row size kv_rank + rot_dim, a window ring if `window` is set.
A sequence that starts at position 0 attends over the step's own rows; one that goes on (by
one token or many) stores first and attends over the cache.

A call that reads another call's cache (`shares_kv`) has no down projection and no latent norm: it projects
and rotates its own queries and attends, with its own W_uk and W_uv, over the rows that the other call has
stored (this step's rows among them), every row over the cache.  The other call's kv_rank, rot_dim and
rotation are this one's.
"""
from __future__ import annotations

import functools
import math
from typing import List, Mapping, Optional

import torch

from .. import ops
from ..errors import KernelError, SpecError
from ..registry import part_impl, register_part
from . import linear
from .base import CallStore, KVNeed, Mixer, StepInfo, WeightSpec


# From so many rows that start at position 0 on their keys and values are formed, if there are also PROMPT_WORK numbers of
# latents: what the absorbed form pays grows with the rank, the formed one's walk does not.  Measured, absorbed / formed: eight
# layers of Nuvivik (rank 512) with 64 rows 1.03 / 0.97 ms, 128 rows 1.24 / 1.12, 512 rows 2.36 / 1.67, 4,000 rows 19.3 / 7.1; one
# layer's attention at 256 rows with rank 512, 256 and 128: 69 / 51, 43 / 37 and 37 / 43 us; at 1,024 rows with rank 24: 161 / 53.
PROMPT_ROWS = 64
PROMPT_WORK = 64 * 512


@functools.lru_cache(maxsize=256)
def key_shares(rows: int, heads: int, rank: int, keys: int, fill: float, sms: int) -> int:
    """The shares that the keys of `rows` single rows are cut into, eight heads to a block and one block to an SM: those with the least
    estimated time, and of near ties the most (a replayed step's rows grow beyond what its launches were planned with).  `keys`: the most that a row sees; `fill`: what the rows see over rows x keys.
    The estimate, us: a block takes 3.0 and 2.55 a tile of 32 keys; blocks that do not run at once come in rounds, whole ones where the rows
    are alike, as SMs come free where they are not; a merge takes 5.1, 0.16 a share, and its way through memory.  Fitted to rows of 512 + 64 numbers
    (B200, 1 to 128 rows of 8, 16 and 32 heads, 300 to 4,096 keys; deviation 6%).  Against the best of all shares, as many as run at once take
    1.14 times as long on average over 159 such batches, shares that fill the GPU twice 1.12 times and these 1.01; us, in that order:
    8 rows of 300 to 1,024 keys 21.5 / 26 / 21, 33 of 1,024 51 / 65 / 51, 48 of 1,024 89 / 82 / 72, 40 of 64 to 4,096 330 / 118 / 100."""
    tiles = -(-keys // 32)
    groups = (heads + 7) // 8
    costs = {}
    for shares in range(1, min(32, (keys + 63) // 64) + 1):
        more = max(0.0, rows * groups * shares / sms - 1.0)             # rounds after the first
        rounds = fill * math.ceil(more) + (1.0 - fill) * more
        cost = 3.0 + 2.55 * -(-tiles // shares) + rounds * (3.0 + 2.55 * max(1.0, fill * tiles / shares))
        if shares > 1:
            cost += 5.1 + 0.16 * shares + 0.024 * rows * shares * heads * rank / 8192
        costs[shares] = cost
    near = 1.02 * min(costs.values())
    return max(shares for shares, cost in costs.items() if cost <= near)


class LatentAttention(Mixer):
    graph_safe = True
    # bfloat16 rows whose sizes fit run the MMA kernel (the 32-bit query and weights as two bfloat16 terms each);
    # False keeps the FMA kernel everywhere (tests compare the two)
    use_tensor_cores = True

    def __init__(self, spec, rt):
        super().__init__(spec, rt)
        p = spec.params
        self.width = int(p["width"])
        self.n_heads = int(p["n_heads"])
        self.dim = int(p["dim"])                  # unrotated query/key numbers per head
        self.rot_dim = int(p["rot_dim"])          # rotated ones
        self.vdim = int(p["vdim"])
        self.rank = int(p["kv_rank"])
        self.scale = float(p["scale"])
        self.eps = float(p["eps"])
        self.window: Optional[int] = p.get("window")
        self.has_sink = bool(p.get("sink", False))
        self.shares_kv = bool(p.get("shares_kv", False))
        self.q_rank = int(p.get("q_rank") or 0)   # 0: queries straight from the layer's input
        if self.shares_kv and self.window:
            raise SpecError("arch spec error: a latent attention that reads another call's cache keeps no window of its own")
        pos_spec = p.get("position")
        self.position = part_impl("position", pos_spec.kind)(pos_spec, rt) if pos_spec else None
        if min(self.n_heads, self.dim, self.rot_dim, self.vdim, self.rank) <= 0 or self.q_rank < 0:
            raise SpecError("arch spec error: latent attention needs positive sizes")
        self.q_cols = self.n_heads * (self.dim + self.rot_dim)
        self.row = self.rank + self.rot_dim

    def weight_specs(self) -> List[WeightSpec]:
        w = self.spec.weights
        if self.q_rank:
            out = [WeightSpec(w["dq"], (self.q_rank, self.width), "matrix", 0.02),
                   WeightSpec(w["dq_norm"], (self.q_rank,), "vector", 0.1),
                   WeightSpec(w["uq"], (self.q_cols, self.q_rank), "matrix", 0.05)]
        else:
            out = [WeightSpec(w["q"], (self.q_cols, self.width), "matrix", 0.02)]
        if not self.shares_kv:
            out += [WeightSpec(w["dkv"], (self.row, self.width), "matrix", 0.02),
                    WeightSpec(w["dkv_norm"], (self.rank,), "vector", 0.1)]
        out += [WeightSpec(w["uk"], (self.n_heads * self.dim, self.rank), "matrix", 0.05),
               WeightSpec(w["uv"], (self.n_heads * self.vdim, self.rank), "matrix", 0.05),
               WeightSpec(w["o"], (self.width, self.n_heads * self.vdim), "matrix", 0.02)]
        if self.has_sink:
            out.append(WeightSpec(w["sink"], (self.n_heads,), "vector", 0.5))
        return out

    def bind(self, tensors: Mapping[str, torch.Tensor]) -> None:
        w = self.spec.weights
        q = self._matrix(tensors[w["dq" if self.q_rank else "q"]])
        self.q_norm = self._vector32(tensors[w["dq_norm"]]) if self.q_rank else None
        self.w_uq = linear.pad_rows(self._matrix(tensors[w["uq"]])) if self.q_rank else None
        self.w_norm = None
        if self.shares_kv:
            self.w_in = q
        else:
            dkv = self._matrix(tensors[w["dkv"]])
            if q.dtype != dkv.dtype:
                q, dkv = q.float(), dkv.float()
            self.w_in = torch.cat([q, dkv], dim=0).contiguous()          # one product for q and the down projection
            self.w_norm = self._vector32(tensors[w["dkv_norm"]])
        if self.q_rank:
            self.w_in = linear.pad_rows(self.w_in)
        uk = self._matrix(tensors[w["uk"]]).view(self.n_heads, self.dim, self.rank)
        self.w_uk_t = uk.transpose(1, 2).contiguous()                # [heads, rank, dim]: q'_h = W_uk_h^T q_h
        self.w_uv = self._matrix(tensors[w["uv"]]).view(self.n_heads, self.vdim, self.rank).contiguous()
        # a prompt's keys and values as one product of its latent rows [c | rotated part]: the heads' W_uk, then their W_uv,
        # with zeros under the rotated part
        self.w_expand = None
        if self._prompt_sizes_fit() and uk.dtype == torch.bfloat16 and self.w_uv.dtype == torch.bfloat16:
            both = torch.cat([uk.reshape(-1, self.rank), self.w_uv.reshape(-1, self.rank)])
            self.w_expand = torch.cat([both, both.new_zeros((both.shape[0], self.rot_dim))], dim=1).contiguous()
        self.w_o = self._matrix(tensors[w["o"]])
        self.sink = self._vector32(tensors[w["sink"]]) if self.has_sink else None

    def kv_need(self) -> KVNeed:
        return KVNeed(1, self.row, self.window, keys_only=True)

    def plan(self, rows: int, step: StepInfo):
        """(shares of the keys, rows per block) for `rows` rows of a step.  Rows of one sequence that follow one another
        share the keys they read: four to a block (prompts, long pieces).  Few rows, or rows of different sequences
        (decoding), run one to a block, and their keys are cut into shares: see key_shares where an SM holds one block, and
        where it holds several, shares that fill the GPU about twice; at least two tiles of 32 keys per share, at most 32 shares."""
        if not step.single_token and rows >= 64:
            return 1, 4
        blocks = rows * ((self.n_heads + 7) // 8)
        sms = ops.sm_count()
        longest = step.max_len_after
        keys = min(int(self.window), longest) if self.window else longest
        rot_dims = self.position.kernel_args()[1] if self.position else 0
        if self.use_tensor_cores and not self.rt.is_fp32 and ops.latent_attn_blocks(self.rank, self.row, rot_dims) == 1:
            live = min(rows, step.max_live) if step.max_live else rows
            return key_shares(live, self.n_heads, self.rank, keys, step.fill_for(self.window), sms), 1
        return max(1, min(32, (keys + 63) // 64, (2 * sms + blocks - 1) // blocks)), 1

    def _prompt_sizes_fit(self) -> bool:
        """Whether a prompt's keys and values may be formed and walked over by the tcgen05 kernel (csrc/latent_prompt.cu)."""
        sizes = (self.dim, self.rot_dim, self.vdim)
        return (not self.rt.is_fp32 and not self.shares_kv and self.scale > 0 and self.rank % 8 == 0 and
                all(n % 8 == 0 and n <= most for n, most in zip(sizes, ops.LATENT_PROMPT_SIZES)))

    def forward(self, h: torch.Tensor, step: StepInfo, store: CallStore) -> torch.Tensor:
        return self._run(h, step, store, False)

    def forward_partial(self, h: torch.Tensor, step: StepInfo, store: CallStore) -> torch.Tensor:
        """As forward, but the output projection may come back as float32 partial sums [parts, N, width] for a consumer
        that adds them."""
        return self._run(h, step, store, True)

    def _run(self, h: torch.Tensor, step: StepInfo, store: CallStore, partial_ok: bool) -> torch.Tensor:
        n = h.shape[0]
        cache = store.kv
        if cache is None or store.owns_kv == self.shares_kv:
            raise KernelError("latent attention: the call's cache and the mixer's tensors do not fit (a mixer without a "
                              "down projection reads another call's cache, and only such a mixer does)")
        H, R, D = self.n_heads, self.rank, self.row
        proj = linear.matmul(h, self.w_in)
        kc = None if self.shares_kv else torch.empty((n, D), dtype=h.dtype, device=h.device)
        inv_freq, rot_dims, style = self.position.kernel_args() if self.position else (None, 0, 1)
        q_first = self.q_rank or self.q_cols                # the column where the down projection's part of `proj` begins
        parts = {} if self.shares_kv else dict(down=(proj, q_first), w_norm=self.w_norm, kc=kc, cache=cache)
        q = proj
        if self.q_rank:
            cq = torch.empty((n, self.q_rank), dtype=h.dtype, device=h.device)
            parts.update(cq=(proj, 0), cq_norm=self.q_norm, cq_out=cq)
        if parts:
            ops.latent_prep(step, R, self.rot_dim, self.eps, inv_freq, rot_dims, style, **parts)
        if self.q_rank:
            q = linear.matmul(cq, self.w_uq)
        att = torch.empty((n, H * self.vdim), dtype=h.dtype, device=h.device)
        nf = 0 if self.shares_kv else (n if step.from_zero else step.fresh_tokens)
        done = 0
        if nf >= PROMPT_ROWS and nf * R >= PROMPT_WORK and self.w_expand is not None and self.use_tensor_cores and not step.single_token:
            kv = linear.matmul(kc[:nf], self.w_expand, out_dtype=torch.float32)
            ops.latent_prompt(q, self.dim, self.vdim, inv_freq, rot_dims, style, kv, kc, self.sink, att, step, nf, R, self.scale,
                              self.window)
            done = nf
        if done < n:
            self._run_absorbed(q, kc, att, done, nf, step, cache, (inv_freq, rot_dims, style))
        return linear.matmul_or_partials(att, self.w_o) if partial_ok else linear.matmul(att, self.w_o)

    def _run_absorbed(self, q, kc, att, first: int, nf: int, step: StepInfo, cache, rot) -> None:
        """Rows first .. of `att` from the queries taken to the latent: rows up to nf attend over the step's own latent
        rows kc, the others over the cache."""
        n, H, R = q.shape[0], self.n_heads, self.rank
        q_lat = torch.empty((n, H, R), dtype=torch.float32, device=q.device)
        o_lat = torch.empty((n, H, R), dtype=q.dtype, device=q.device)      # what the value expansion reads
        # q'_h = W_uk_h^T q_h
        ops.heads_product(q, first * q.shape[1], q.shape[1], self.dim + self.rot_dim, self.w_uk_t, q_lat, first * H * R, H * R, R, n - first)
        attend = functools.partial(ops.latent_attn, q_lat, q, self.dim, *rot)
        if nf > first:
            shares, per_block = self.plan(nf, step)
            attend(kc, None, self.sink, o_lat, step, 0, nf, R, self.scale, self.window, paged=False,
                   n_splits=shares, rows_per_block=per_block, tensor_cores=self.use_tensor_cores)
        if nf < n:
            if cache.ring_pages > 0 and not step.replayed:
                room = cache.ring_pages * ops.PAGE_TOKENS - int(self.window) + 1
                news = [step.cu_host[i + 1] - step.cu_host[i] for i in range(step.fresh_seqs, step.n_seqs)] if step.cu_host else []
                if news and max(news) > room:
                    raise KernelError(f"a step that continues sequences brings {max(news)} tokens to a layer that keeps "
                                      f"a window of {self.window} keys in a ring of {cache.ring_pages * ops.PAGE_TOKENS}: "
                                      f"at most {room} fit")
            rows = n - nf
            shares, per_block = self.plan(rows, step)
            attend(None, cache, self.sink, o_lat, step, nf, rows, R, self.scale, self.window, paged=True,
                   n_splits=shares, rows_per_block=per_block, tensor_cores=self.use_tensor_cores)
        ops.heads_product(o_lat, first * H * R, H * R, R, self.w_uv, att, first * H * self.vdim, H * self.vdim, self.vdim, n - first)


register_part("mixer", "latent_attention", LatentAttention)
