"""Kernels that a rule on sizes picks between, at sizes on either side of its lines that the tests of the kernels themselves do not
reach: the checks are theirs."""
import pytest
import torch

import test_gpu_row_words as rows
import test_gpu_state_step as state
import test_gpu_top_k_bound as top_k

pytestmark = pytest.mark.gpu
both = pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])


@both
@pytest.mark.parametrize("columns,parts,T", [(132, 2, 739), (132, 2, 741), (256, 1, 1481), (1024, 2, 745), (1020, 8, 186), (8, 1, 3)])
def test_gated_norm(dtype, columns, parts, T):
    rows.test_gated_norm_in_parts(dtype, columns, parts, T)


@both
@pytest.mark.parametrize("H,G,N,P,taps,lens", [(12, 2, 128, 64, 4, [1] * 190), (12, 2, 128, 64, 4, [180]), (12, 2, 128, 64, 4, [1, 300, 2, 1000]),
                                               (4, 1, 64, 64, 2, [1043, 3]), (6, 1, 64, 64, 3, [2500]), (24, 2, 128, 64, 3, [3, 1, 117])])
def test_state_space_rows(dtype, H, G, N, P, taps, lens):
    rows.test_state_space_rows(dtype, H, G, N, P, taps, lens)


@both
@pytest.mark.parametrize("H,d,dv,rot,interleaved", [(2, 128, 128, 64, False), (4, 64, 64, 64, True), (3, 128, 8, 128, True), (4, 48, 96, 32, False)])
def test_retention_rows(dtype, H, d, dv, rot, interleaved):
    rows.test_retention_rows(dtype, H, d, dv, rot, interleaved)


@pytest.mark.parametrize("d,rot", [(112, 16), (120, 120), (128, 128), (256, 64)])
def test_chunked_attention_rows(d, rot):
    rows.test_chunked_attention_rows_rotated_in_pairs(d, rot)


@pytest.mark.parametrize("form", ["head", "delta", "channel", "token", "delta_head"])
@pytest.mark.parametrize("n,H,d,dv", [(1, 8, 128, 128), (2, 8, 128, 128), (4, 2, 256, 256), (1, 2, 256, 256), (1, 4, 192, 128), (3, 2, 33, 16),
                                      (2, 2, 32, 16), (600, 2, 72, 16), (300, 2, 72, 16), (70, 1, 64, 28)])
def test_single_tokens(form, n, H, d, dv):
    state.test_single_tokens(form, [1] * n, H, H, d, dv)


@pytest.mark.parametrize("k", [640, 641, 1000])
@pytest.mark.parametrize("vocab", [40000, 100000, 131072, 140000])
def test_kept_ids(vocab, k):
    top_k.test_kept_ids(vocab, k)


@pytest.mark.parametrize("rows_,experts,width,tokens", [(1, 16, 1024, 149), (2, 130, 1028, 148), (1, 130, 64, 400), (1, 130, 64, 600), (2, 64, 64, 400)])
@pytest.mark.parametrize("given", [False, True])
def test_route(rows_, experts, width, tokens, given):
    """Every form of the routing kernel: deep and plain loads, one warp a token and sixteen."""
    from cpp_minilamma_b200.csrc import kernels as K
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(experts + tokens)
    top = 4
    h = torch.randn((tokens, width), generator=gen, device=dev).to((torch.float32, torch.bfloat16)[rows_ - 1])
    w = torch.randn((experts, width), generator=gen, device=dev) / width ** 0.5
    z = h.double() @ w.double().T
    chosen = torch.full((tokens, top), -1, dtype=torch.int32, device=dev)
    weight = torch.zeros((tokens, top), device=dev)
    K.moe_route(h, w, None, chosen, weight, top, logits=z.float() if given else None)
    best = z.topk(top + 1, dim=1)
    clear = (best.values[:, :-1] - best.values[:, 1:]).min(1).values > 1e-4  # float32 sums of `width` terms of a few tell them apart
    assert clear.float().mean() > 0.9
    assert torch.equal(chosen[clear].long(), best.indices[clear][:, :top])
    assert (weight.double() - best.values[:, :top].softmax(1))[clear].abs().max() <= 1e-5


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("per,experts,width,inter,top", [(0.25, 16, 512, 1024, 4), (0.6, 16, 512, 2048, 4), (3, 16, 520, 2048, 4), (1, 64, 256, 1408, 6), (4, 4, 64, 64, 2),
                                                         (170, 4, 72, 136, 1), (300, 3, 512, 264, 2)])
def test_small_and_wide_tiles(per, experts, width, inter, top, form):
    """gate_up's 16-row tiles in long and in short stages and tiles of 128 rows, against float64 of the same bfloat16 values."""
    from cpp_minilamma_b200.csrc import kernels as K
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(experts + width)
    draw = lambda *shape: torch.randn(shape, generator=gen, device=dev)
    T = max(1, round(per * experts / top))
    chosen = torch.stack([torch.randperm(experts, generator=gen, device=dev)[:top] for _ in range(T)]).int().contiguous()
    h = draw(T, width).to(torch.bfloat16)
    first = (0.2 * draw(experts, inter * (1 if form else 2), width)).to(torch.bfloat16)
    down, weight = (0.2 * draw(experts, width, inter)).to(torch.bfloat16), torch.rand((T, top), generator=gen, device=dev)
    n = T * top
    tile = K.moe_tile_rows(True, n, experts, width, inter)
    assert tile == (16 if per < 100 else 128)
    tiles = K.moe_max_tiles(n, experts, tile)
    ints = lambda count: torch.full((count,), -7, dtype=torch.int32, device=dev)
    plan = K.MoePlan(ints(n), ints(experts + 1), ints(tiles), ints(tiles), ints(1), tile, True)
    K.moe_sort(chosen, plan, experts)
    act = torch.full((n, inter), 7.0, dtype=torch.bfloat16, device=dev)
    y = torch.full((n, width), 7.0, device=dev)
    K.moe_gate_up(h, first, act, plan, top, form=form)
    K.moe_down(act, down, y, weight, plan, top)
    order = plan.order.long()
    expert = chosen.view(-1)[order].long()
    for e in expert.unique().tolist():
        at = (expert == e).nonzero()[:, 0]
        x, w = h[order[at] // top].double(), first[e].double()
        z, slack = x @ w.T, (x.abs() @ w.abs().T) * width ** 0.5 * 2.0 ** -23  # float32 sums of `width` terms
        if form:
            want, slack = torch.nn.functional.gelu(z), 1.2 * slack
        else:
            gate, up = z[:, :inter], z[:, inter:]
            want = torch.nn.functional.silu(gate) * up
            slack = 1.2 * slack[:, :inter] * up.abs() + gate.abs() * slack[:, inter:]
        assert ((act[at].double() - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-6).all(), e
        a, d = act[at].double(), down[e].double()
        want = weight.view(-1)[order[at]].double()[:, None] * (a @ d.T)
        assert ((y[order[at]].double() - want).abs() <= (a.abs() @ d.abs().T) * inter ** 0.5 * 2.0 ** -23 + 1e-6).all(), e
