"""The recurrences of steps that bring every sequence one token, all five forms, at the edges of the kernel's tiles: fewer rows
than a thread's or a block's, rows that are no multiple of either, value columns around 64, several heads on one key head;
and tokens spread unevenly over the sequences.  Against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["head", "delta", "channel", "token", "delta_head"])
@pytest.mark.parametrize("lens,H,G,d,dv", [
    ([1, 1, 1], 2, 1, 4, 4), ([1] * 5, 3, 3, 21, 100), ([1, 1], 2, 2, 32, 64), ([1, 0, 2], 4, 2, 36, 68), ([1], 1, 1, 64, 60),
    ([1, 1, 1], 4, 4, 66, 128), ([3, 0, 0, 1], 2, 1, 128, 128), ([1, 1], 2, 2, 128, 256), ([1, 1], 2, 1, 131, 24),
    ([1] * 3, 2, 2, 256, 64), ([1, 1], 2, 2, 48, 30), ([1, 1], 1, 1, 260, 8)])  # the last two: left to the general scan
def test_single_tokens(form, lens, H, G, d, dv):
    from cpp_minilamma_b200.csrc import kernels as K
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(sum(lens) * 31 + d + dv)
    T, n = sum(lens), len(lens)
    draw = lambda *shape: torch.randn(shape, generator=gen, device=dev)
    unit = lambda *shape: torch.rand(shape, generator=gen, device=dev)
    q, k, v = draw(T, G * d), draw(T, G * d) / d ** 0.5, draw(T, H * dv)
    channel, delta = form in ("delta", "channel"), form in ("delta", "delta_head")
    g = 0.5 + 0.5 * unit(T, H * d) if channel else None
    token = 0.5 + 0.5 * unit(T, H) if form in ("token", "delta_head") else None
    head = 0.5 + 0.5 * unit(H) if form == "head" else None
    beta = unit(T, H) if delta else None
    state = draw(n + 1, H, d, dv)
    slots = list(range(n, 0, -1))
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    starts = [sum(lens[:i]) for i in range(n)]
    want_s, want_o = state.double().clone(), torch.zeros((T, H, dv), dtype=torch.float64, device=dev)
    for i in range(n):
        for t in range(starts[i], starts[i] + lens[i]):
            for h in range(H):
                S = want_s[slots[i], h]
                kh, qh = (z[t].double().view(G, d)[h // (H // G)] for z in (k, q))
                vh = v[t].double().view(H, dv)[h]
                S = S * (g[t].double().view(H, d)[h][:, None] if channel else token[t, h].double() if token is not None else head[h].double())
                u = beta[t, h].double() * (vh - S.T @ kh) if delta else vh
                S = S + torch.outer(kh, u)
                want_s[slots[i], h] = S
                want_o[t, h] = S.T @ qh
    out = torch.full((T, H * dv), 7.0, device=dev)
    K.state_scan(q, k, v, g, beta, head, state, out, ints(slots), ints(starts), ints(lens), n, H, G, d, dv, token_decay=token)
    torch.cuda.synchronize()
    # float32 sums of d terms of the size of a few, twice over (S^T k enters u, which enters the output)
    bound = 4 * d ** 0.5 * 2.0 ** -23
    assert (out.double().view(T, H, dv) - want_o).abs().max() <= bound * max(1.0, want_o.abs().max().item())
    assert (state.double() - want_s).abs().max() <= bound * max(1.0, want_s.abs().max().item())


@pytest.mark.parametrize("form", ["head", "delta", "channel", "token", "delta_head"])
@pytest.mark.parametrize("d", [32, 64, 128, 256])
def test_no_further_off_than_the_general_scan(form, d):
    """Outputs' and states' distance to 64 bits as root mean squares over 16,384 outputs, beside the general scan's (which a row more than
    there are sequences calls for).  A tenth of slack: two such means of the same size differ by a few parts in a hundred."""
    from cpp_minilamma_b200.csrc import kernels as K
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(d)
    n, H, dv = 4, 64, 64
    draw = lambda *shape: torch.randn(shape, generator=gen, device=dev)
    unit = lambda *shape: torch.rand(shape, generator=gen, device=dev)
    q, k, v = draw(n + 1, H * d) / d, draw(n + 1, H * d) / d ** 0.5, draw(n + 1, H * dv)
    channel, delta = form in ("delta", "channel"), form in ("delta", "delta_head")
    g = 0.5 + 0.5 * unit(n + 1, H * d) if channel else None
    token = 0.5 + 0.5 * unit(n + 1, H) if form in ("token", "delta_head") else None
    head = 0.5 + 0.5 * unit(H) if form == "head" else None
    beta = unit(n + 1, H) if delta else None
    before = draw(n, H, d, dv)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    decay = (g[:n].double().view(n, H, d, 1) if channel else token[:n].double().view(n, H, 1, 1) if token is not None
             else head.double().view(1, H, 1, 1))
    S = before.double() * decay
    kd, qd, vd = (x[:n].double().view(n, H, -1) for x in (k, q, v))
    u = beta[:n].double()[..., None] * (vd - torch.einsum("nhkv,nhk->nhv", S, kd)) if delta else vd
    S = S + kd[..., None] * u[:, :, None]
    want = torch.einsum("nhkv,nhk->nhv", S, qd)
    squares = []
    for rows in (n, n + 1):
        state, out = before.clone(), torch.zeros((rows, H * dv), device=dev)
        cut = lambda x: None if x is None else x[:rows].contiguous()
        K.state_scan(cut(q), cut(k), cut(v), cut(g), cut(beta), head, state, out, ints(list(range(n))), ints(list(range(n))), ints([1] * n),
                     n, H, H, d, dv, token_decay=cut(token))
        squares.append([(out[:n].double().view(n, H, dv) - want).square().mean().sqrt().item(), (state.double() - S).square().mean().sqrt().item()])
    assert squares[0][0] <= 1.1 * squares[1][0] and squares[0][1] <= 1.1 * squares[1][1], squares
