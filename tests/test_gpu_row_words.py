"""The kernels that prepare rows for the state mixers and chunked attention, where they work on words of several columns and
walks of several tokens: rotations in halves and in pairs over all or some of a head's words, sequences that begin and end
inside a walk, parts of a row from one word to the widest that a warp holds and one more.  Against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _turned(x, rot, interleaved, c, s):
    out = x.clone()
    a, b = (slice(0, rot, 2), slice(1, rot, 2)) if interleaved else (slice(0, rot // 2), slice(rot // 2, rot))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


def _tables(rot, gen):
    angle = torch.rand((128, max(rot // 2, 1)), generator=gen, device=DEV) * 6.0
    return angle.cos().contiguous(), angle.sin().contiguous()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,d,dv,rot,interleaved", [(2, 16, 8, 16, False), (3, 48, 24, 32, False), (2, 128, 256, 128, False), (2, 24, 8, 8, True),
                                                    (1, 8, 8, 8, True), (4, 64, 32, 40, True), (2, 24, 8, 24, False), (2, 16, 12, 4, True),
                                                    (2, 16, 8, 0, False)])
def test_retention_rows(dtype, H, d, dv, rot, interleaved):
    from cpp_minilamma_b200.csrc import kernels as K
    gen = torch.Generator(device=DEV).manual_seed(H * d + rot)
    T, n = 9, H * d
    proj = torch.randn((T, 2 * n + H * dv + 8), generator=gen, device=DEV).to(dtype)
    pos = torch.randint(0, 128, (T,), generator=gen, device=DEV, dtype=torch.int32)
    cos, sin = _tables(rot, gen)
    q, k, v = (torch.full((T, w), 7.0, device=DEV) for w in (n, n, H * dv))
    K.retention_prepare(proj, cos if rot else None, sin if rot else None, pos, q, k, v, H, d, dv, rot, interleaved, 0.3)
    c, s = (z[pos.long()].double()[:, None] for z in (cos, sin))
    for got, at, scale in ((q, 0, 1.0), (k, n, 0.3)):
        x = proj[:, at:at + n].double().view(T, H, d)
        want = (_turned(x, rot, interleaved, c, s) if rot else x) * scale
        assert (got.double().view(T, H, d) - want).abs().max() <= 4 * 2.0 ** -24 * x.abs().max()
    assert torch.equal(v, proj[:, 2 * n:2 * n + H * dv].float())


@pytest.mark.parametrize("d,rot", [(16, 16), (64, 24), (128, 64), (24, 8), (32, 4)])
def test_chunked_attention_rows_rotated_in_pairs(d, rot):
    from cpp_minilamma_b200.csrc import kernels as K
    gen = torch.Generator(device=DEV).manual_seed(d + rot)
    H, G, dv, T = 4, 2, 16, 5
    qkv = torch.randn((T, (H + G) * d + G * dv), generator=gen, device=DEV).to(torch.bfloat16)
    qw, kw = (1 + 0.2 * torch.randn((n * d,), generator=gen, device=DEV) for n in (H, G))
    cos, sin = _tables(rot, gen)
    pos = torch.tensor([0, 63, 64, 100, 7], dtype=torch.int32, device=DEV)
    ints = torch.arange(T, dtype=torch.int32, device=DEV)
    table = torch.arange(2 * T, dtype=torch.int32, device=DEV).view(T, 2).contiguous()
    q = torch.zeros((T, H * d), dtype=torch.bfloat16, device=DEV)
    kc, vc = (torch.zeros((2 * T, G, 64, w), dtype=torch.bfloat16, device=DEV) for w in (d, dv))
    K.local_attention_prepare(qkv, qw, kw, cos, sin, pos, ints, ints, table, q, kc, vc, H, G, d, dv, rot, True, 1e-5)
    for t in range(T):
        p = int(pos[t])
        for got, at, n, w in ((q[t], 0, H, qw), (kc[int(table[t, p // 64]), :, p % 64].reshape(-1), H * d, G, kw)):
            x = qkv[t, at:at + n * d].double()
            x = (x / (x.square().mean() + 1e-5).sqrt() * w.double()).view(n, d)
            want = _turned(x, rot, True, cos[p].double(), sin[p].double()).reshape(-1)
            assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()
        assert torch.equal(vc[int(table[t, p // 64]), :, p % 64].reshape(-1), qkv[t, (H + G) * d:])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,N,P,taps,lens", [(2, 1, 8, 8, 4, [1, 2, 700, 3, 9]), (4, 2, 16, 24, 3, [610]), (3, 3, 24, 8, 2, [300, 300, 1]),
                                               (130, 1, 8, 8, 4, [5, 1, 1, 8])])
def test_state_space_rows(dtype, H, G, N, P, taps, lens):
    from cpp_minilamma_b200.csrc import kernels as K
    gen = torch.Generator(device=DEV).manual_seed(H + taps)
    draw = lambda *shape: torch.randn(shape, generator=gen, device=DEV)
    inner, gn, T, n = H * P, G * N, sum(lens), len(lens)
    C = inner + 2 * gn
    proj = draw(T, (2 * inner + 2 * gn + H + 7) // 8 * 8).to(dtype)
    w, b, a_log, bias, state = 0.6 * draw(C, taps), 0.3 * draw(C), draw(H) - 0.5, draw(H), draw(n + 1, taps - 1, C)
    slots = list(range(n, 0, -1))
    starts = [sum(lens[:i]) for i in range(n)]
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    q, k, u, xs, decay = (torch.full((T, width), 7.0, device=DEV) for width in (gn, gn, inner, inner, H))
    K.ssd_prepare(proj, w, b, state, a_log, bias, ints([i for i, m in enumerate(lens) for _ in range(m)]), ints(slots), ints(starts),
                  q, k, u, xs, decay, H, G, N, P, taps)
    for i, m in enumerate(lens):
        rows = slice(starts[i], starts[i] + m)
        x = torch.cat([state[slots[i]].double(), proj[rows, inner:inner + C].double()])
        y = b.double() + sum(x[j:j + m] * w[:, j].double() for j in range(taps))
        y = y * torch.sigmoid(y)
        dt = torch.nn.functional.softplus(proj[rows, inner + C:inner + C + H].double() + bias.double())
        for got, want in ((xs, y[:, :inner]), (u, y[:, :inner] * dt.repeat_interleave(P, 1)), (k, y[:, inner:inner + gn]),
                          (q, y[:, inner + gn:]), (decay, torch.exp(-a_log.double().exp() * dt))):
            # sums of `taps` terms of a few, softplus and two exponentials in float32
            assert (got[rows].double() - want).abs().max() <= 5e-6 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("columns,parts,T", [(4, 3, 5), (60, 2, 3), (128, 8, 40), (132, 1, 2), (512, 8, 700), (1024, 2, 3), (1028, 1, 2)])
def test_gated_norm_in_parts(dtype, columns, parts, T):
    from cpp_minilamma_b200.csrc import kernels as K
    gen = torch.Generator(device=DEV).manual_seed(columns + parts)
    draw = lambda *shape: torch.randn(shape, generator=gen, device=DEV)
    width = columns * parts
    o, xs, skip, weight = draw(T, width), draw(T, width), draw(width // 4), 1 + 0.3 * draw(width)
    gate = draw(T, width + 8).to(dtype)
    for x in (xs, None):
        out = torch.full((T, width), 7.0, device=DEV).to(dtype)
        K.gated_group_norm(o, x, skip if x is not None else None, gate, weight, out, 4, parts, 1e-5)
        y = o.double() if x is None else o.double() + skip.double().repeat_interleave(4) * x.double()
        y = (y * torch.nn.functional.silu(gate[:, :width].double())).view(T, parts, columns)
        want = (y / (y.square().mean(-1, keepdim=True) + 1e-5).sqrt()).view(T, width) * weight.double()
        rounding = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21
        assert ((out.double() - want).abs() <= rounding * want.abs() + 1e-5).all()
