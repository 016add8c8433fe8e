"""The float32 product for the few rows of a decode step at the edges of its launch: every batch width it is built for and one
more row, weight rows that leave a warp's four unfilled, K below and beyond a run of 128 and its remainders, every split of
K, the bias and the gated epilogue.  Against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(1, 4), (5, 124), (16, 128), (33, 132), (192, 512), (1039, 192), (96, 2048), (2048, 8196)])
def test_product(rows, n, k):
    from cpp_minilamma_b200.csrc import kernels as K
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(rows * 1000 + n + k)
    draw = lambda *shape: torch.randn(shape, generator=gen, device=dev)
    x, w, bias = draw(rows, k), draw(n, k), draw(n)
    assert K.linear_f32_supported(x, w)
    # float32 sums of k terms, and the bias's addition
    slack = (x.abs().double() @ w.abs().double().T) * k ** 0.5 * 2.0 ** -24 + 1e-7 * bias.abs()
    want = x.double() @ w.double().T
    for slices in (0, 1, 2, 4, 8):
        for b in (None, bias):
            out = torch.full((rows, n), 7.0, device=dev)
            K.linear_f32(x, w, b, out, slices=slices)
            exact = want if b is None else want + b
            assert ((out.double() - exact).abs() <= slack + exact.abs() * 2.0 ** -23).all(), (slices, b is None)
    for epilogue in ((K.EPI_SWIGLU, K.EPI_GEGLU) if n % 16 == 0 else ()):
        assert K.linear_f32_supported(x, w, epilogue)
        blocks = want.view(rows, n // 16, 2, 8)
        gate, up = blocks[:, :, 0].reshape(rows, -1), blocks[:, :, 1].reshape(rows, -1)
        s = slack.view(rows, n // 16, 2, 8)
        # silu is 1.1-Lipschitz and gelu (tanh form) 1.13; both are no larger than their argument
        bound = 1.2 * s[:, :, 0].reshape(rows, -1) * up.abs() + gate.abs() * s[:, :, 1].reshape(rows, -1)
        if epilogue == K.EPI_SWIGLU:
            exact, own = torch.nn.functional.silu(gate) * up, 0.0
        else:
            # formed as g sigmoid(y): y is rounded by no more than 2^-22 |y|, and |y| times sigmoid's slope stays below 0.28
            exact, own = torch.nn.functional.gelu(gate, approximate="tanh") * up, 2.0 ** -23 * (gate * up).abs()
        for slices in (0, 1, 2, 4, 8):
            out = torch.full((rows, n // 2), 7.0, device=dev)
            K.linear_f32(x, w, None, out, epilogue, slices)
            assert ((out.double() - exact).abs() <= bound + own + exact.abs() * 2.0 ** -20).all(), (epilogue, slices)


def test_refused_and_left_to_the_library():
    from cpp_minilamma_b200.csrc import kernels as K
    dev = torch.device("cuda:0")
    w = torch.zeros(32, 64, device=dev)
    assert not K.linear_f32_supported(torch.zeros(17, 64, device=dev), w)
    assert not K.linear_f32_supported(torch.zeros(2, 66, device=dev)[:, 2:], w)  # rows with a stride of their own
    assert not K.linear_f32_supported(torch.zeros(2 * 64 + 1, device=dev)[1:].view(2, 64), w)  # off the 16-byte boundary
    assert not K.linear_f32_supported(torch.zeros(2, 62, device=dev), torch.zeros(32, 62, device=dev))
    assert not K.linear_f32_supported(torch.zeros(2, 64, device=dev), torch.zeros(24, 64, device=dev), K.EPI_SWIGLU)
    with pytest.raises(K.KernelError):
        K.linear_f32(torch.zeros(2, 64, device=dev), w, None, torch.zeros(2, 31, device=dev))


@pytest.mark.parametrize("m,n,k,own", [(4, 16384, 64, True), (5, 16384, 64, False), (8, 4096, 64, True), (8, 4100, 252, False), (8, 4100, 256, True),
                                       (9, 64, 124, False), (9, 64, 128, True), (16, 4100, 252, False), (16, 12288, 256, True), (16, 12292, 256, False),
                                       (16, 12292, 2048, True), (17, 64, 256, False)])
def test_left_to_the_library_where_that_is_faster(m, n, k, own):
    from types import SimpleNamespace
    from cpp_minilamma_b200.csrc import kernels as K
    from cpp_minilamma_b200.parts.linear import Linear
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(m + n + k)
    x, w, bias = (torch.randn(s, generator=gen, device=dev) for s in ((m, k), (n, k), (n,)))
    assert K.linear_f32_pays(x, w) == own
    part, before = Linear(w, "w", bias=bias), K.calls.get("linear_f32", 0)
    out = part._product_f32(SimpleNamespace(small_rows=64), x, torch.empty((m, n), device=dev))
    assert K.calls.get("linear_f32", 0) - before == own
    want = x.double() @ w.double().T + bias
    # float32 sums of k terms, and the bias's addition
    slack = (x.abs().double() @ w.abs().double().T) * k ** 0.5 * 2.0 ** -24 + 1e-7 * bias.abs() + want.abs() * 2.0 ** -23
    assert ((out.double() - want).abs() <= slack).all()
