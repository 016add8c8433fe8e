"""The routed products of prompts (tcgen05, pairs of multiprocessors) at the edges of their tiles: rows of an expert around
128 and 256, one row and none, widths that are no multiple of the 64 columns of a stage or of a tile's 256 columns, more
tiles than pairs, and an expert that gets nearly every row; both forms.  Against float64 of the same bfloat16 values."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("counts,width,inter", [
    ([1], 64, 64), ([0, 3, 0, 2], 72, 40), ([127, 128, 129], 192, 136), ([255, 256, 257, 0, 1], 520, 264),
    ([400, 30, 513], 8, 8), ([600, 1, 700, 300], 1024, 1032), ([40] * 24, 136, 2048)])
def test_routed_products(counts, width, inter, form):
    from cpp_minilamma_b200.csrc import kernels as K
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(sum(counts) + width)
    draw = lambda *shape: torch.randn(shape, generator=gen, device=dev)
    top, E = 2, len(counts)
    of = torch.cat([torch.full((n,), e, dtype=torch.int32, device=dev) for e, n in enumerate(counts)])
    if of.numel() % top:
        of = torch.cat([of, of[-1:]])
    n_pairs = of.numel()
    chosen = of[torch.randperm(n_pairs, generator=gen, device=dev)].view(-1, top).contiguous()
    h = draw(n_pairs // top, width).to(torch.bfloat16)
    first = (0.2 * draw(E, inter * (1 if form else 2), width)).to(torch.bfloat16)
    down = (0.2 * draw(E, width, inter)).to(torch.bfloat16)
    weight = torch.rand((n_pairs // top, top), generator=gen, device=dev)
    rows = K.moe_tile_rows(True, 1 << 30, 1)
    tiles = K.moe_max_tiles(n_pairs, E, rows)
    ints = lambda n: torch.full((n,), -7, dtype=torch.int32, device=dev)
    plan = K.MoePlan(ints(n_pairs), ints(E + 1), ints(tiles), ints(tiles), ints(1), rows, True)
    assert K.moe_needs_rows(plan)
    K.moe_sort(chosen, plan, E)
    act = torch.full((n_pairs, inter), 7.0, dtype=torch.bfloat16, device=dev)
    y = torch.full((n_pairs, width), 7.0, dtype=torch.float32, device=dev)
    K.moe_gate_up(h, first, act, plan, top, form=form)
    K.moe_down(act, down, y, weight, plan, top)
    torch.cuda.synchronize()
    assert K.take_device_error() == 0
    order = plan.order.long()
    expert = chosen.view(-1)[order].long()
    for e in range(E):
        at = (expert == e).nonzero()[:, 0]
        if at.numel() == 0:
            continue
        x, w = h[order[at] // top].double(), first[e].double()
        z, terms = x @ w.T, x.abs() @ w.abs().T
        slack = terms * width ** 0.5 * 2.0 ** -23  # float32 sums of `width` terms
        if form:
            want, slack = torch.nn.functional.gelu(z), 1.2 * slack
        else:  # silu is 1.1-Lipschitz and no larger than its argument
            gate, up = z[:, :inter], z[:, inter:]
            want = torch.nn.functional.silu(gate) * up
            slack = 1.2 * slack[:, :inter] * up.abs() + gate.abs() * slack[:, inter:]
        # one rounding to bfloat16 and a hardware exponential (2 ulp of float32) in front of it
        assert ((act[at].double() - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-6).all(), (e, form)
        a, d = act[at].double(), down[e].double()
        want = weight.view(-1)[order[at]].double()[:, None] * (a @ d.T)
        slack = (a.abs() @ d.abs().T) * inter ** 0.5 * 2.0 ** -23
        assert ((y[order[at]].double() - want).abs() <= slack + 1e-6).all(), (e, form)


@pytest.mark.parametrize("width", [8, 64, 5 * 64, 6 * 64, 6 * 64 + 8, 13 * 64])
def test_back_to_back(width):
    """Launches on each other's heels, with fewer, as many and more fills of the ring than it has stages: the pairs leave with
    nothing on its way into their shared memory, so that every launch finds what the first found."""
    from cpp_minilamma_b200.csrc import kernels as K
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(width)
    draw = lambda *shape: torch.randn(shape, generator=gen, device=dev)
    E, inter, n_pairs = 3, 256, 400
    chosen = torch.randint(0, E, (n_pairs, 1), generator=gen, device=dev, dtype=torch.int32)
    h, first = draw(n_pairs, width).to(torch.bfloat16), (0.2 * draw(E, 2 * inter, width)).to(torch.bfloat16)
    down, weight = (0.2 * draw(E, inter, width)).to(torch.bfloat16), torch.rand((n_pairs, 1), generator=gen, device=dev)
    rows = K.moe_tile_rows(True, 1 << 30, 1)
    tiles = K.moe_max_tiles(n_pairs, E, rows)
    ints = lambda n: torch.zeros(n, dtype=torch.int32, device=dev)
    plan = K.MoePlan(ints(n_pairs), ints(E + 1), ints(tiles), ints(tiles), ints(1), rows, True)
    K.moe_sort(chosen, plan, E)
    act = torch.empty((40, n_pairs, inter), dtype=torch.bfloat16, device=dev)
    y = torch.empty((40, n_pairs, inter), dtype=torch.float32, device=dev)
    room = torch.empty_like(h)
    for i in range(40):
        K.moe_gate_up(h, first, act[i], plan, 1, rows=room)
        K.moe_down(h, down, y[i], weight, plan, 1)  # any rows in the experts' order do
    torch.cuda.synchronize()
    assert K.take_device_error() == 0
    assert (act == act[:1]).all() and (y == y[:1]).all()
    assert torch.isfinite(y).all() and y.abs().max() > 0
