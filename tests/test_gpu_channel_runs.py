"""The delta rule with a decay per key channel, a run of tokens at a time: runs that end at, before and behind a block of 8 and a
run of 32, several heads on one key head, sizes below and at the kernel's paddings, decays from 1 down to 0 (a channel that
forgets everything at once, and one that forgets within a few tokens), from a state and twice in a row.  Against float64, as
is the token-by-token scan beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _reference(q, k, v, g, beta, S, share):
    out = torch.empty(v.shape, dtype=torch.float64)
    for t in range(q.shape[0]):
        S = g[t][:, :, None] * S
        kt, qt = k[t][share], q[t][share]
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, kt))
        S = S + kt[:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", S, qt)
    return out, S


@pytest.mark.parametrize("strong", [False, True])
@pytest.mark.parametrize("H,G,d,dv,lens", [(2, 2, 128, 128, [257, 3]), (2, 1, 64, 64, [70, 1, 33]), (3, 3, 32, 128, [300]), (1, 1, 16, 16, [64]),
                                           (2, 2, 12, 20, [90]), (4, 2, 128, 32, [7, 8, 9, 31, 32]), (2, 1, 100, 36, [65, 40]),
                                           (1, 1, 4, 4, [25, 24, 17, 16, 15])])
def test_channel_delta_in_runs(H, G, d, dv, lens, strong):
    from cpp_minilamma_b200.csrc import kernels as K
    gen = torch.Generator().manual_seed(d + dv + len(lens))
    n_seqs, share, T = len(lens), torch.arange(H) // (H // G), sum(lens)
    state = torch.randn((n_seqs + 1, H, d, dv), generator=gen).to(DEV)
    before = state.cpu().double()
    slots = list(range(n_seqs))[::-1]
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    runs = [(i, row0) for i, n in enumerate(lens) for row0 in range(0, n, K.STATE_RUN)]
    first_run = [next(j for j, (s, _) in enumerate(runs) if s == i) for i in range(n_seqs)]
    starts = [sum(lens[:i]) for i in range(n_seqs)]
    flat = lambda x: x.reshape(T, -1).contiguous().to(DEV)
    for turn in range(2):
        unit = lambda x: x / x.norm(dim=-1, keepdim=True)
        q, k = unit(torch.randn((T, G, d), generator=gen)) / d ** 0.5, unit(torch.randn((T, G, d), generator=gen))
        k[1::3] = k[0:len(k[1::3]) * 3:3]
        v, beta = torch.randn((T, H, dv), generator=gen), torch.sigmoid(2 * torch.randn((T, H), generator=gen))
        log_g = -torch.exp((3.0 if strong else 1.5) * torch.randn((T, H, d), generator=gen) - (0.0 if strong else 3.0))
        log_g[::5] = 0.0
        if strong:
            log_g[3::11, :, ::2] = -200.0
        g = torch.exp(log_g)
        out = torch.full((T, H * dv), float("nan"), device=DEV)
        scratch = torch.full((K.state_chunks_scratch(len(runs), H, d, dv, True, True),), float("nan"), device=DEV)
        walked, walked_out = state.clone(), torch.empty_like(out)
        K.state_scan(flat(q), flat(k), flat(v), flat(g), flat(beta), None, walked, walked_out, ints(slots), ints(starts), ints(lens),
                     n_seqs, H, G, d, dv)
        K.state_chunks(flat(q), flat(k), flat(v), state, out, scratch, ints([s for s, _ in runs]), ints([r for _, r in runs]),
                       ints(first_run), ints(slots), ints(starts), ints(lens), n_seqs, H, G, d, dv, beta=flat(beta),
                       channel_decay=flat(g))
        for i, (s, n) in enumerate(zip(slots, lens)):
            rows = slice(starts[i], starts[i] + n)
            want, after = _reference(q[rows].double(), k[rows].double(), v[rows].double(), g[rows].double(), beta[rows].double(),
                                     before[s], share)
            scale = max(1.0, want.abs().max().item())
            for kind, (o, S) in enumerate(((out, state), (walked_out, walked))):
                err = (o[rows].cpu().double().view(n, H, dv) - want)
                # float32 sums of d and of 32 terms, handed from run to run (as the other recurrences in runs are held to)
                assert err.abs().max().item() <= 2e-5 * scale, (kind, turn, i)
                assert (S[s].cpu().double() - after).abs().max().item() <= 2e-5 * max(1.0, after.abs().max().item()), (kind, turn, i)
            before[s] = after
        assert torch.equal(state[n_seqs].cpu().double(), before[n_seqs])
        before = state.cpu().double()


@pytest.mark.parametrize("strong", [False, True])
@pytest.mark.parametrize("H,d,dv,lens", [(16, 128, 128, [257]), (8, 64, 64, [100, 64, 200]), (16, 32, 64, [300, 90])])
def test_no_further_off_than_token_by_token(H, d, dv, lens, strong):
    """The outputs' and the states' distance to 64 bits, as root mean squares over all heads, beside the scan's that the runs stand
    in for.  A tenth of slack: two such means of the same size differ by a few parts in a hundred."""
    from cpp_minilamma_b200.csrc import kernels as K
    gen = torch.Generator().manual_seed(d + dv)
    n_seqs, T = len(lens), sum(lens)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    runs = [(i, row0) for i, n in enumerate(lens) for row0 in range(0, n, K.STATE_RUN)]
    first = [next(j for j, (s, _) in enumerate(runs) if s == i) for i in range(n_seqs)]
    starts = [sum(lens[:i]) for i in range(n_seqs)]
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k = unit(torch.randn((T, H, d), generator=gen)) / d ** 0.5, unit(torch.randn((T, H, d), generator=gen))
    v, beta = torch.randn((T, H, dv), generator=gen), torch.sigmoid(2 * torch.randn((T, H), generator=gen))
    g = torch.exp(-torch.exp((3.0 if strong else 1.5) * torch.randn((T, H, d), generator=gen) - (0.0 if strong else 3.0)))
    state = (0.1 * torch.randn((n_seqs, H, d, dv), generator=gen)).to(DEV)
    flat = lambda x: x.reshape(T, -1).contiguous().to(DEV)
    walked, out, walked_out = state.clone(), torch.empty((T, H * dv), device=DEV), torch.empty((T, H * dv), device=DEV)
    before = state.cpu().double()
    lists = (ints(list(range(n_seqs))), ints(starts), ints(lens), n_seqs, H, H, d, dv)
    K.state_scan(flat(q), flat(k), flat(v), flat(g), flat(beta), None, walked, walked_out, *lists)
    scratch = torch.empty(K.state_chunks_scratch(len(runs), H, d, dv, True, True), device=DEV)
    K.state_chunks(flat(q), flat(k), flat(v), state, out, scratch, ints([s for s, _ in runs]), ints([r for _, r in runs]), ints(first),
                   *lists, beta=flat(beta), channel_decay=flat(g))
    squares = torch.zeros((2, 2), dtype=torch.float64)
    for i, n in enumerate(lens):
        rows = slice(starts[i], starts[i] + n)
        want, after = _reference(q[rows].double(), k[rows].double(), v[rows].double(), g[rows].double(), beta[rows].double(), before[i],
                                 torch.arange(H))
        for kind, (o, S) in enumerate(((out, state), (walked_out, walked))):
            squares[0, kind] += (o[rows].cpu().double().view(n, H, dv) - want).square().sum()
            squares[1, kind] += (S[i].cpu().double() - after).square().sum()
    assert (squares[:, 0].sqrt() <= 1.1 * squares[:, 1].sqrt()).all(), squares.sqrt()


def test_refused():
    from cpp_minilamma_b200.csrc import kernels as K
    z = lambda *shape: torch.zeros(shape, device=DEV)
    i = torch.zeros(1, dtype=torch.int32, device=DEV)
    with pytest.raises(K.KernelError):  # a decay per channel without the delta rule
        K.state_chunks(z(4, 8), z(4, 8), z(4, 8), z(1, 1, 8, 8), z(4, 8), z(99999), i, i, i, i, i, i, 1, 1, 1, 8, 8, channel_decay=z(4, 8))


@pytest.mark.parametrize("form", ["head", "token", "delta_head", "delta"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_later_tokens_stay_out_of_earlier_ones(form, bad):
    """A value that is not finite reaches its own token and those behind it, as token by token: not the earlier tokens of its
    run, nor another head or sequence; and where nothing follows it, the state is infinite where it is token by token."""
    from cpp_minilamma_b200.csrc import kernels as K
    H, d, dv, lens, at = 2, 64, 36, [83, 40], [43, 83 + 39]  # inside a block of 8 of the second run; the last token of all
    gen = torch.Generator().manual_seed(7)
    T, n_seqs = sum(lens), len(lens)
    draw = lambda *shape: torch.randn(shape, generator=gen).to(DEV)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    q, k, v = draw(T, H * d) / d ** 0.5, draw(T, H * d) / d ** 0.5, draw(T, H * dv)
    for t in at:
        v[t, 5] = bad  # head 0
    unit = lambda *shape: 0.5 + 0.5 * torch.rand(shape, generator=gen).to(DEV)
    channel = unit(T, H * d) if form == "delta" else None
    token = unit(T, H) if form in ("token", "delta_head") else None
    head = unit(H) if form == "head" else None
    beta = unit(T, H) if form in ("delta", "delta_head") else None
    runs = [(i, row0) for i, n in enumerate(lens) for row0 in range(0, n, K.STATE_RUN)]
    first = [next(j for j, (s, _) in enumerate(runs) if s == i) for i in range(n_seqs)]
    state = draw(n_seqs, H, d, dv)
    walked, out, walked_out = state.clone(), torch.empty((T, H * dv), device=DEV), torch.empty((T, H * dv), device=DEV)
    lists = (ints([0, 1]), ints([0, lens[0]]), ints(lens), n_seqs, H, H, d, dv)
    K.state_scan(q, k, v, channel, beta, head, walked, walked_out, *lists, token_decay=token)
    scratch = torch.full((K.state_chunks_scratch(len(runs), H, d, dv, beta is not None, channel is not None),), float("nan"), device=DEV)
    K.state_chunks(q, k, v, state, out, scratch, ints([s for s, _ in runs]), ints([r for _, r in runs]), ints(first), *lists,
                   head_decay=head, token_decay=token, beta=beta, channel_decay=channel)
    ok = torch.isfinite(walked_out)
    assert not ok.all() and ok[:at[0]].all() and ok[83:at[1]].all()
    assert torch.equal(torch.isfinite(out), ok)
    assert (out - walked_out)[ok].abs().max() <= 4e-5 * walked_out[ok].abs().max()  # two float32 sums, 2e-5 each
    assert torch.equal(torch.isfinite(state), torch.isfinite(walked))
    assert torch.equal(torch.isnan(state[1]), torch.isnan(walked[1]))
