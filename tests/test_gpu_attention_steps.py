"""The tcgen05 prompt attention at its two head sizes: walks of one, two and an odd number of pages, tiles that end inside them,
and every mask the kernel knows, over contexts whose last page is full, nearly full and nearly empty.  The cache holds
not-a-numbers wherever no sequence has a position.  Against float64 of the same bfloat16 values."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("masks", [{}, {"window": 100}, {"window": 70, "keep_first": 5}, {"window": 64, "keep_first": 130}, {"chunk": 96},
                                   {"chunk": 128}, {"softcap": 3.0}, {"sink": True}, {"sink_values": True}, {"gate": True},
                                   {"window": 90, "softcap": 2.0, "sink": True}])
@pytest.mark.parametrize("H,G", [(4, 2), (3, 1)])
@pytest.mark.parametrize("d", [64, 128])
def test_masks_and_partial_pages(masks, H, G, d):
    from cpp_minilamma_b200.csrc import kernels as K
    PAGE = 64
    gen = torch.Generator(device=DEV).manual_seed(H + len(masks))
    draw = lambda *shape: torch.randn(shape, generator=gen, device=DEV)
    lens = [1, 63, 64, 65, 128, 129, 200, 3, 300, 1, 130]
    ctx = [1, 63, 64, 65, 128, 129, 200, 66, 449, 192, 257]
    n, T = len(lens), sum(lens)
    pages = [-(-c // PAGE) for c in ctx]
    order = torch.randperm(sum(pages), generator=gen, device=DEV).cpu().tolist()
    table = torch.full((n, max(pages) + 1), 10 ** 6, dtype=torch.int32)
    kc, vc = (torch.full((sum(pages), G, PAGE, d), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    keys, values = [], []
    for i, c in enumerate(ctx):
        k, v = draw(c, G, d).to(torch.bfloat16), draw(c, G, d).to(torch.bfloat16)
        keys.append(k.double())
        values.append(v.double())
        for j in range(pages[i]):
            page = order.pop()
            table[i, j] = page
            part = slice(j * PAGE, min(c, (j + 1) * PAGE))
            kc[page, :, :part.stop - part.start] = k[part].transpose(0, 1)
            vc[page, :, :part.stop - part.start] = v[part].transpose(0, 1)
    q = (2 * draw(T, H, d)).to(torch.bfloat16)
    starts = [sum(lens[:i]) for i in range(n)]
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    tiles = [(i, r) for i, m in enumerate(lens) for r in range(0, m, 64)]
    wide = [(i, r) for i, m in enumerate(lens) for r in range(0, m, 128)]
    extra = dict(masks)
    window = extra.pop("window", 0)
    sink_values = draw(H) if extra.pop("sink_values", None) else None
    gates = draw(T, H + 8).to(torch.bfloat16) if extra.pop("gate", None) else None
    scale = d ** -0.5
    out = torch.full((T, H * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    K.attention_prefill(q.view(T, H * d), kc, vc, ints(list(range(n))), ints(ctx), ints(starts), ints(lens), ints([t for t, _ in tiles]),
                        ints([r for _, r in tiles]), table.to(DEV), out, len(tiles), H, G, d, window, scale,
                        wide_tiles=(ints([t for t, _ in wide]), ints([r for _, r in wide])), sink_values=sink_values,
                        gate=(gates, 3) if gates is not None else None, **extra)
    torch.cuda.synchronize()
    assert K.take_device_error() == 0
    for i, (m, c) in enumerate(zip(lens, ctx)):
        rows = slice(starts[i], starts[i] + m)
        at, j = torch.arange(c - m, c, device=DEV)[:, None], torch.arange(c, device=DEV)[None]
        seen = j <= at
        if window:
            seen = seen & ((j > at - window) | (j < masks.get("keep_first", 0)))
        if masks.get("chunk"):
            seen = seen & (j // masks["chunk"] == at // masks["chunk"])
        share = torch.arange(H, device=DEV) // (H // G)
        s = torch.einsum("thd,jhd->htj", q[rows].double(), keys[i][:, share]) * scale
        if masks.get("softcap"):
            s = masks["softcap"] * torch.tanh(s / masks["softcap"])
        s = s.masked_fill(~seen, -torch.inf)
        if masks.get("sink") or sink_values is not None:
            sink = (sink_values.double() if sink_values is not None else torch.zeros(H, device=DEV).double())[:, None, None].expand(-1, m, 1)
            p = torch.cat([s, sink], -1).softmax(-1)[..., :-1]
        else:
            p = s.softmax(-1)
        want = torch.einsum("htj,jhd->thd", p, values[i][:, share])
        # P is rounded to 8 bits against a sum of the unrounded: 2^-8 of the weighted values' sizes; and the result's rounding
        bound = 2.0 ** -8 * torch.einsum("htj,jhd->thd", p, values[i][:, share].abs()) + 2.0 ** -8 * want.abs() + 1e-4
        if gates is not None:
            g = torch.sigmoid(gates[rows, 3:3 + H].double())[..., None]
            want, bound = want * g, bound * g + 1e-4
        got = out[rows].double().view(m, H, d)
        assert ((got - want).abs() <= bound).all(), (i, (got - want).abs().max().item())
