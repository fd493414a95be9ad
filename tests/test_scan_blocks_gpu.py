"""The recurrence over blocks of 32 tokens against float64: decays of every size, corrections, head sizes that are padded, entries
on the edges of a block, and what is not finite."""

import math

import pytest
import torch

from test_recurrent_kernels_gpu import DEV, _batch

pytestmark = pytest.mark.gpu


def exact(q, k, v, decay, beta, bonus, state, lengths, heads, dim, vdim):
    """``decay [T, heads, dim]``; everything float64; the read-outs and the final states as the kernels lay them out."""
    out, final, at = [], [], 0
    for e, n in enumerate(lengths):
        S = state[e].view(heads, vdim, dim).transpose(1, 2).clone()
        for t in range(at, at + n):
            qt, kt, vt = q[t].view(heads, dim), k[t].view(heads, dim), v[t].view(heads, vdim)
            if bonus is not None:
                pair = kt[:, :, None] * vt[:, None, :]
                out.append(torch.einsum("hk,hkv->hv", qt, S + bonus[:, :, None] * pair))
                S = S * decay[t][:, :, None] + pair
                continue
            S = S * decay[t][:, :, None]
            u = vt if beta is None else beta[t][:, None] * (vt - torch.einsum("hk,hkv->hv", kt, S))
            S = S + kt[:, :, None] * u[:, None, :]
            out.append(torch.einsum("hk,hkv->hv", qt, S))
        final.append(S.transpose(1, 2).reshape(-1))
        at += n
    return torch.stack(out).view(at, heads * vdim), torch.stack(final)


def given(kind, decays, heads, dim, vdim, lengths):
    tokens = sum(lengths)
    generator = torch.Generator(device=DEV).manual_seed(dim + len(lengths))
    draw = lambda *shape: torch.randn(*shape, generator=generator, device=DEV)      # noqa: E731
    q, k = draw(tokens, heads * dim) * dim ** -0.5, draw(tokens, heads, dim)
    k = (k / k.norm(dim=-1, keepdim=True)).view(tokens, -1).contiguous()
    rate = torch.rand(tokens, heads * dim, generator=generator, device=DEV)
    # near one, where the products span a wide range, and as small as they come (zeros among them: what was before is forgotten)
    decay = {"slow": 1 - 0.05 * rate, "fast": rate * 0.9 + 0.05, "zeros": rate * (rate > 0.3)}[decays]
    options = {}
    if kind == "delta":
        options["beta"] = torch.rand(tokens, heads, generator=generator, device=DEV)
    elif kind == "bonus":
        options["bonus"] = draw(heads, dim)
    return q, k, draw(tokens, heads * vdim), decay.contiguous(), options, draw(len(lengths), heads * dim * vdim) * 0.3


def take(q, k, v, decay, options, state, lengths, heads, dim, vdim, in_blocks):
    from rapid_llm_b200.engine.batch import Workspace
    from rapid_llm_b200.ops import kernels

    batch = _batch(lengths, list(range(len(lengths))), [5] * len(lengths))
    batch.max_query_len = max(lengths)
    out, after = torch.empty_like(v), state.clone()
    kernels.linear_scan(q, k, v, decay, out, after, batch, heads=heads, kv_heads=heads, dim=dim, vdim=vdim,
                        pieces=Workspace(sum(lengths), torch.device(DEV)) if in_blocks else None, blocks_from=in_blocks, **options)
    assert int(batch.fault.item()) == 0
    return out, after


@pytest.mark.parametrize("decays", ["slow", "fast", "zeros"])
@pytest.mark.parametrize("kind,heads,dim,vdim", [("delta", 3, 64, 64), ("delta", 2, 36, 44), ("delta", 2, 128, 128), ("delta", 2, 100, 132),
                                                 ("plain", 2, 128, 128), ("plain", 2, 100, 132), ("bonus", 2, 128, 128), ("bonus", 2, 68, 36)])
def test_blocks_are_as_near_as_the_walk(kind, decays, heads, dim, vdim):
    first = 64
    lengths = [first, first + 1, first + 31, 4 * first + 33]
    q, k, v, decay, options, state = given(kind, decays, heads, dim, vdim, lengths)
    doubled = {name: t.double() for name, t in options.items()}
    want, final = exact(q.double(), k.double(), v.double(), decay.double().view(-1, heads, dim), doubled.get("beta"), doubled.get("bonus"),
                        state.double(), lengths, heads, dim, vdim)
    off = []
    for in_blocks in (0, first):
        out, after = take(q, k, v, decay, options, state, lengths, heads, dim, vdim, in_blocks)
        off.append((float((out.double() - want).norm() / want.norm()), float((after.double() - final).norm() / final.norm())))
    (walked, walked_state), (read, left) = off
    # a mean over ten thousand roundings and more on each side; where a state forgets at once both are a few roundings: a number of
    # a block's record is rounded three times (a product of decays, what it multiplies, U), 2^-24 each at most, where a walk
    # multiplies once
    assert read <= 1.1 * walked + 2.0 ** -24 and left <= 1.1 * walked_state + 2.0 ** -24, off
    if decays == "slow":      # what engines' decays are like: nearer than the walk
        assert read <= walked and left <= walked_state, off


@pytest.mark.parametrize("kind", ["plain", "bonus", "delta"])
def test_what_is_not_finite_reaches_no_earlier_token_and_no_other_column(kind):
    heads, dim, vdim, at = 2, 128, 64, 77
    lengths = [160]
    q, k, v, decay, options, state = given(kind, "slow", heads, dim, vdim, lengths)
    clean, after = take(q, k, v, decay, options, state, lengths, heads, dim, vdim, 64)
    v[at, 5] = math.inf
    v[at + 3, 9] = math.nan
    out, odd = take(q, k, v, decay, options, state, lengths, heads, dim, vdim, 64)
    touched = torch.zeros_like(out, dtype=torch.bool)
    touched[at:, 5], touched[at + 3 :, 9] = True, True
    # (sums behind the tokens before are formed one after the other there: another order, 32 roundings)
    size = clean.abs().max()
    assert bool(((out - clean).abs()[~touched] <= 32 * 2.0 ** -23 * size).all())
    assert not bool(torch.isfinite(out[at + 4 :, [5, 9]]).any())
    columns = torch.ones(heads, vdim, dtype=torch.bool, device=DEV)
    columns[0, [5, 9]] = False
    kept = columns[:, :, None].expand(heads, vdim, dim).reshape(-1)
    assert bool(((odd - after).abs()[0, kept] <= 64 * 2.0 ** -23 * after.abs().max()).all())
