"""The float32 product on the tensor cores (csrc/gemm_f32.cu): against float64, bits of a row alone and among others in every
tile width, rows that start inside a word, operands that are not finite."""
import pytest
import torch

from vosti_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def status():
    return torch.zeros(1, dtype=torch.int32, device=DEV)


def draw(seed, rows, n, k):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(rows, k, generator=gen, device=DEV), torch.randn(n, k, generator=gen, device=DEV)


def bound(x, w):
    """Per output, over the sum of magnitudes: a rounding of the running sum per 64 k and K segment, at most four truncations (two
    roundings' worth each) of a 64-k sum, 7 K / 16 truncations of sums 2^-6 as large (two terms below 2^-7), and the term left out: l is
    below 2^-15 of its operand, so l l is below 2^-30, a fraction of one rounding."""
    k = x.shape[1]
    steps = -(-k // 64) + 8 + 2 * 4 + 2 * (7 * k / 16) * 2.0 ** -6 + 1
    return steps * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)


# rows around the widths of the token tiles, n and k around 128 and 64, one to eight K segments
@pytest.mark.parametrize("rows,n,k", [(1, 16, 128), (32, 127, 130), (33, 129, 191), (64, 300, 256), (65, 64, 2048), (128, 4100, 513),
                                      (129, 128, 4096), (193, 640, 1027), (257, 257, 640), (385, 25000, 132), (600, 384, 1000)])
def test_against_float64_and_rows_alone(status, rows, n, k):
    x, w = draw(rows + n + k, rows, n, k)
    y = ops.gemm_f32(x, w, status)
    want = x.double() @ w.double().T
    assert bool(((y.double() - want).abs() <= bound(x, w)).all()) and status.item() == 0
    chain = ops.gemm_simt(x, w, status)
    assert (y.double() - want).norm() <= (chain.double() - want).norm()
    for a, b in [(0, 1), (rows // 2, rows // 2 + 1), (0, min(rows, 40)), (max(rows - 70, 0), rows), (0, min(rows, 150)), (0, min(rows, 200))]:
        assert torch.equal(ops.gemm_f32(x[a:b].contiguous(), w, status), y[a:b])
    # the same numbers on places that are not whole words
    xs, ws = torch.empty(rows * k + 1, device=DEV), torch.empty(n * k + 3, device=DEV)
    xs[1:], ws[3:] = x.view(-1), w.view(-1)
    assert torch.equal(ops.gemm_f32(xs[1:].view(rows, k), ws[3:].view(n, k), status), y)


@pytest.mark.parametrize("n,k", [(200, 4096), (4096, 1024), (25000, 1024)])          # eight, four and one K segments
@pytest.mark.parametrize("adjacent", [True, False])
def test_rows_of_few_products_are_as_near_as_the_chain(status, n, k, adjacent):
    """One to sixteen products a row, next to one another or anywhere. With one the result is the product rounded once, as the chain's:
    it may differ by l l (2^-30 of the product, mean 2^-32) and a truncation of the small sum (2^-31) only, 2^-6 of a rounding."""
    for count in (1, 2, 3, 4, 6, 8, 16):
        gen = torch.Generator(device=DEV).manual_seed(count)
        w, x = torch.randn(n, k, generator=gen, device=DEV), torch.zeros(70, k, device=DEV)
        if adjacent:
            places = torch.randint(0, k - count + 1, (70, 1), generator=gen, device=DEV) + torch.arange(count, device=DEV)
        else:
            places = torch.rand(70, k, generator=gen, device=DEV).argsort(1)[:, :count]
        x.scatter_(1, places, torch.randn(70, count, generator=gen, device=DEV))
        want = x.double() @ w.double().T
        error = lambda y: (y.double() - want).norm().item()
        assert error(ops.gemm_f32(x, w, status)) <= (1 + 2.0 ** -6) * error(ops.gemm_simt(x, w, status)), count


def test_positive_sums_and_small_and_large_operands(status):
    x, w = draw(5, 70, 200, 4096)
    for a, b in ((x.abs(), w.abs()), (x * 1e-30, w * 1e3), (x * 1e-25, w * 1e-12), (x * 1e20, w * 1e15)):
        want = a.double() @ b.double().T
        rel = lambda y: ((y.double() - want).norm() / want.norm()).item()
        assert rel(ops.gemm_f32(a, b, status)) <= rel(ops.gemm_simt(a, b, status))


@pytest.mark.parametrize("rows,n,k", [(70, 200, 2048), (130, 20000, 1024), (20, 4096, 1024)])         # eight, one and four K segments
@pytest.mark.parametrize("a,b", [(-70, -70), (-75, -68), (-105, 60), (-110, 60), (-118, 60), (-122, 70), (-130, 90), (-140, 100), (-126, 10),
                                 (70, -122), (100, -140), (31, -112)])
def test_operands_whose_last_bits_no_term_holds(status, rows, n, k, a, b):
    """A third of the rows of x times 2^a, a half of w's times 2^b: the error of each of the four blocks is no larger than the chain's, a row
    alone has the same bits, and zeros stay zeros."""
    x, w = draw(rows + k, rows, n, k)
    x[::3], w[::2] = (x[::3].double() * 2.0 ** a).float(), (w[::2].double() * 2.0 ** b).float()
    x[4] = 0
    want = x.double() @ w.double().T
    y, chain = ops.gemm_f32(x, w, status), ops.gemm_simt(x, w, status)
    third, odd = torch.arange(rows, device=DEV) % 3 == 0, torch.arange(n, device=DEV) % 2 == 0
    for i in (third, ~third):
        for j in (odd, ~odd):
            error = lambda t: (t.double() - want)[i][:, j].norm().item()
            assert error(y) <= error(chain), (error(y), error(chain))
    assert not y[4].any() and status.item() == 0
    for t in (0, 1):
        assert torch.equal(ops.gemm_f32(x[t:t + 1], w, status)[0], y[t])


def test_operands_that_are_not_finite(status):
    x, w = draw(6, 40, 200, 512)
    x[3, 7], x[5, 9], x[6, :], w[10, 3], x[7, 11], w[:, 11] = float("inf"), float("nan"), -3.4028234e38, float("-inf"), 3.4028e38, 0.25
    y, chain = ops.gemm_f32(x, w, status), ops.gemm_simt(x, w, status)
    assert torch.equal(torch.isnan(y), torch.isnan(chain)) and torch.equal(torch.isinf(y), torch.isinf(chain))
    finite = torch.isfinite(chain)
    assert torch.allclose(y[finite], chain[finite], rtol=1e-4, atol=1e-4)
