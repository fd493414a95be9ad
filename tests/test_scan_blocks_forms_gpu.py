"""What the recurrence over blocks of tokens accepts, in one step as an engine makes them: every kind of decay, scaled and skipped
values, shared keys, rows off a 16-byte boundary, short entries beside long ones, entries from zeros and from a carried state."""

from types import SimpleNamespace

import pytest
import torch

from test_recurrent_kernels_gpu import DEV, _batch

pytestmark = pytest.mark.gpu

FIRST = 64
LENGTHS, STARTS, SLOTS = [1, FIRST - 1, FIRST, 3 * FIRST + 5, 2], [8, 0, 0, 40, 3], [4, 1, 0, 3, 2]


def step(form, heads, kv_heads, dim, vdim, off=0):
    """Inputs of a step; ``off``: floats by which rows and values miss a 16-byte boundary."""
    tokens = sum(LENGTHS)
    generator = torch.Generator(device=DEV).manual_seed(dim + heads)
    draw = lambda *shape: torch.randn(*shape, generator=generator, device=DEV)      # noqa: E731
    near_one = lambda *shape: 1 - 0.1 * torch.rand(*shape, generator=generator, device=DEV)      # noqa: E731

    def rows(values):
        wide = torch.full((tokens, values.shape[1] + (off or 4)), 7.0, device=DEV)
        wide[:, off : off + values.shape[1]] = values
        return wide[:, off : off + values.shape[1]]

    k = torch.nn.functional.normalize(draw(tokens, kv_heads, dim), dim=-1).view(tokens, -1)
    case = SimpleNamespace(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, q=rows(draw(tokens, kv_heads * dim) * dim ** -0.5), k=rows(k),
                           v=rows(draw(tokens, heads * vdim)), state=draw(len(LENGTHS), heads * dim * vdim) * 0.3, options={})
    if form == "fixed":
        case.decay = near_one(heads)
    elif form == "per_token":
        case.decay = near_one(tokens, heads)
        case.options = {"v_scale": torch.rand(tokens, heads, generator=generator, device=DEV), "skip": draw(heads)}
    else:
        case.decay = near_one(tokens, heads * dim)
    if form == "bonus":
        case.options = {"bonus": draw(heads, dim)}
    elif form == "delta":
        case.options = {"beta": torch.rand(tokens, heads, generator=generator, device=DEV)}
    elif form == "delta_fixed":
        case.decay = near_one(heads)
        case.options = {"beta": torch.rand(tokens, heads, generator=generator, device=DEV), "skip": draw(heads)}
    return case


def take(case, in_blocks, entries=None):
    """Read-outs and states of ``entries`` (all), in their order in the step."""
    from rapid_llm_b200.engine.batch import Workspace
    from rapid_llm_b200.ops import kernels

    at = [sum(LENGTHS[:e]) for e in range(len(LENGTHS))]
    entries = list(range(len(LENGTHS))) if entries is None else entries
    index = torch.cat([torch.arange(at[e], at[e] + LENGTHS[e], device=DEV) for e in entries])
    whole = len(entries) == len(LENGTHS)
    part = lambda t: t if whole or t.shape[0] != sum(LENGTHS) else t[index].contiguous()      # noqa: E731
    batch = _batch([LENGTHS[e] for e in entries], [SLOTS[e] for e in entries], [STARTS[e] for e in entries])
    batch.max_query_len = max(LENGTHS[e] for e in entries)
    tokens = len(index)
    wide, state = torch.full((tokens, case.heads * case.vdim + 4), 7.0, device=DEV), case.state.clone()
    out = wide[:, : case.heads * case.vdim]
    kernels.linear_scan(part(case.q), part(case.k), part(case.v), part(case.decay), out, state, batch, heads=case.heads, kv_heads=case.kv_heads,
                        dim=case.dim, vdim=case.vdim, pieces=Workspace(tokens, torch.device(DEV)) if in_blocks else None, blocks_from=in_blocks,
                        **{name: part(t) for name, t in case.options.items()})
    assert int(batch.fault.item()) == 0 and bool((wide[:, case.heads * case.vdim :] == 7.0).all())
    return out, state[[SLOTS[e] for e in entries]]


def exact(case):
    heads, dim, vdim = case.heads, case.dim, case.vdim
    o = {name: t.double() for name, t in case.options.items()}
    out, final, at = [], [], 0
    for e, n in enumerate(LENGTHS):
        S = case.state[SLOTS[e]].double().view(heads, vdim, dim).transpose(1, 2) * float(STARTS[e] > 0)
        for t in range(at, at + n):
            per = lambda x: x[t].double().view(case.kv_heads, dim).repeat_interleave(heads // case.kv_heads, dim=0)      # noqa: E731
            q, k, v = per(case.q), per(case.k), case.v[t].double().view(heads, vdim)
            g = case.decay.double()
            g = g.view(heads, 1, 1) if g.dim() == 1 else g[t].view(heads, -1, 1)
            if "bonus" in o:
                pair = k[:, :, None] * v[:, None, :]
                read = torch.einsum("hk,hkv->hv", q, S + o["bonus"][:, :, None] * pair)
                S = S * g + pair
            else:
                S = S * g
                u = v * o["v_scale"][t][:, None] if "v_scale" in o else v
                if "beta" in o:
                    u = o["beta"][t][:, None] * (v - torch.einsum("hk,hkv->hv", k, S))
                S = S + k[:, :, None] * u[:, None, :]
                read = torch.einsum("hk,hkv->hv", q, S)
            out.append(read + o["skip"][:, None] * v if "skip" in o else read)
        final.append(S.transpose(1, 2).reshape(-1))
        at += n
    return torch.stack(out).view(at, heads * vdim), torch.stack(final)


FORMS = ["fixed", "per_token", "per_row", "bonus", "delta", "delta_fixed"]


@pytest.mark.parametrize("off", [0, 1, 2])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 128, 64), (3, 3, 100, 132), (6, 1, 128, 36)])
def test_a_step_in_every_form(form, heads, kv_heads, dim, vdim, off):
    case = step(form, heads, kv_heads, dim, vdim, off)
    want, final = exact(case)
    away = []
    for in_blocks in (0, FIRST):
        out, state = take(case, in_blocks)
        away.append([float((got.double() - w).norm() / w.norm()) for got, w in ((out, want), (state, final))])
        # and in no entry by itself: a sum of a few dozen numbers that count, each rounded a few times
        assert float((out.double() - want).abs().max()) <= 100 * 2.0 ** -24 * float(want.abs().max())
    (walked, walked_state), (read, left) = away
    # means over ten thousand roundings and more; short entries are walked on both sides
    assert read <= 1.1 * walked and left <= 1.1 * walked_state, away


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 128, 64), (2, 2, 100, 44)])
def test_an_entry_in_blocks_is_the_same_alone_and_beside_others(form, heads, kv_heads, dim, vdim):
    case = step(form, heads, kv_heads, dim, vdim)
    together, states = take(case, FIRST)
    at = 0
    for e, n in enumerate(LENGTHS):
        out, state = take(case, FIRST, [e])
        assert torch.equal(out, together[at : at + n]) and torch.equal(state[0], states[e]), n
        at += n


@pytest.mark.parametrize("form", ["delta", "delta_fixed"])
def test_narrow_heads_with_a_correction(form):
    case = step(form, 4, 2, 64, 64)
    want, final = exact(case)
    (walked, walked_state), (out, state) = take(case, 0), take(case, FIRST)
    assert float((out.double() - want).norm()) <= 1.1 * float((walked.double() - want).norm())
    assert float((state.double() - final).norm()) <= 1.1 * float((walked_state.double() - final).norm())


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("where", ["q", "k", "v", "decay", "state", "strength"])
@pytest.mark.parametrize("form", ["fixed", "per_token", "per_row", "bonus", "delta"])
def test_what_is_not_finite_is_as_the_walk_has_it(form, where, value):
    """Infinities keep their sign and place, what came before and the columns beside stay as they are, and a finite number whose
    leading part rounds to an infinity is a number."""
    case = step(form, 2, 2, 128, 64)
    at = sum(LENGTHS[:3]) + 77           # in the third block of the longest entry
    if where == "state":
        case.state[SLOTS[3], 5 * 128 + 9] = value          # column 5 of head 0
    elif where == "strength":
        name = {"per_token": "v_scale", "delta": "beta", "bonus": "bonus"}.get(form)
        if name is None:
            pytest.skip("values enter as they are")
        case.options[name][(0, 3) if form == "bonus" else (at, 0)] = value
    elif where == "decay":
        if value == 3.4e38:
            pytest.skip("the state overflows at once")
        case.decay[0 if form == "fixed" else (at, 0)] = value
    else:
        getattr(case, where)[at, 3] = value
    if where == "k" and value == 3.4e38:
        pytest.skip("whether a sum behind it overflows is a matter of its order")
    for got, walked in zip(take(case, FIRST), take(case, 0)):
        assert torch.equal(got.isnan(), walked.isnan())
        assert torch.equal(got.isinf(), walked.isinf()) and torch.equal(got[got.isinf()], walked[got.isinf()])
        # the same sums in another order: a few dozen numbers that count, of a size with their column's largest
        shape = (-1, case.heads * case.vdim, case.dim if got.shape[1] > case.heads * case.vdim else 1)
        got, walked, finite = got.reshape(shape), walked.reshape(shape), walked.isfinite().view(shape)
        size = torch.where(finite, walked, 0).abs().amax(dim=(0, 2), keepdim=True).clamp(min=1.0)
        assert bool((((got - walked) / size).abs()[finite] <= 200 * 2.0 ** -24).all())
