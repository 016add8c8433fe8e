"""Prompt attention over a latent on the 5th-generation tensor cores against float64: values are the keys' leading columns.

A weight is rounded to bfloat16 and so is the result: eight significant bits, rounded to nearest, are off by up to 2^-8 of the number (half
of the last place, 2^-7, of a number just above a power of two).  Scores and sums are float32 (2^-12 allows for both)."""
import pytest
import torch

from cpp_minilamma_b200.csrc import kernels as K

pytestmark = pytest.mark.gpu


def _case(lens, starts, heads, row, value, seed):
    """Inputs of a step: the sequences' new tokens behind `starts` earlier ones, pages in a shuffled order, cache rows that no
    sequence has filled with NaN."""
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seed)
    ctx = [a + b for a, b in zip(lens, starts)]
    pages = [-(-c // 64) for c in ctx]
    total = sum(pages) + 3
    order = torch.randperm(total, generator=g, device=dev).tolist()
    table = torch.full((len(lens) + 1, max(pages)), order[-1], dtype=torch.int32)
    cache = torch.full((total, 1, 64, row), float("nan"), device=dev, dtype=torch.bfloat16)
    rows, at = [], 0
    slots = [len(lens) - i for i in range(len(lens))]
    for i, c in enumerate(ctx):
        r = torch.randn((c, row), generator=g, device=dev).bfloat16()
        rows.append(r)
        for p in range(pages[i]):
            page = order[at]
            at += 1
            table[slots[i], p] = page
            part = r[p * 64:(p + 1) * 64]
            cache[page, 0, :part.shape[0]] = part
    q = torch.randn((sum(lens), heads * row), generator=g, device=dev).bfloat16()
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)  # noqa: E731
    starts_of_q = [sum(lens[:i]) for i in range(len(lens))]
    wide = sorted((starts[i] + min(lens[i], r + 128), i, r) for i in range(len(lens)) for r in range(0, lens[i], 128))
    return (q, cache, t(slots), t(ctx), t(starts_of_q), t(lens), t([i for _, i, _ in wide]), t([r for _, _, r in wide]),
            table.to(dev)), rows, starts_of_q


@pytest.mark.parametrize("row,value,window,sink", [(256, 192, 0, None), (256, 256, 0, "zero"), (192, 128, 0, "values"), (256, 200, 100, None),
                                                   (192, 8, 64, "values"), (256, 64, 1, None)])
@pytest.mark.parametrize("lens,starts,heads", [([1], [0], 1), ([128, 129, 2], [0, 0, 63], 3), ([300, 1, 64], [0, 70, 65], 2), ([700], [130], 5)])
def test_against_float64(row, value, window, sink, lens, starts, heads):
    args, rows, q0 = _case(lens, starts, heads, row, value, seed=row + value + sum(lens))
    q = args[0]
    out = torch.full((q.shape[0], heads * value), float("nan"), device=q.device, dtype=torch.bfloat16)
    scale = row ** -0.5
    sinks = torch.linspace(-1.0, 2.0, heads, device=q.device) if sink == "values" else None
    assert K.latent_attention_tc5_supported(q.dtype, row, value)
    K.latent_attention_tiles(*args, out, heads, row, value, window, scale, sink=sink is not None, sink_values=sinks)
    assert K.take_device_error() == 0
    for i, n in enumerate(lens):
        keys = rows[i].double()
        x = q[q0[i]:q0[i] + n].double().view(n, heads, row)
        s = torch.einsum("nhd,td->hnt", x, keys) * scale
        pos = torch.arange(n, device=q.device)[:, None] + starts[i]
        j = torch.arange(keys.shape[0], device=q.device)[None]
        seen = (j <= pos) & ((j > pos - window) if window else True)
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            extra = (sinks.double() if sinks is not None else torch.zeros(heads, device=q.device, dtype=torch.float64))
            s = torch.cat([s, extra[:, None, None].expand(heads, n, 1)], 2)
        p = s.softmax(-1)[:, :, :keys.shape[0]]
        want = torch.einsum("hnt,tv->nhv", p, keys[:, :value])
        size = torch.einsum("hnt,tv->nhv", p, keys[:, :value].abs())
        got = out[q0[i]:q0[i] + n].double().view(n, heads, value)
        bound = (2.0 ** -8 + 2.0 ** -12) * size + 2.0 ** -8 * want.abs() * 1.01 + 1e-6
        assert ((got - want).abs() <= bound).all()


def test_refused():
    for row, value in ((128, 64), (320, 64), (200, 64), (256, 264), (256, 12), (192, 0)):
        assert not K.latent_attention_tc5_supported(torch.bfloat16, row, value)
    assert not K.latent_attention_tc5_supported(torch.float32, 256, 192)
