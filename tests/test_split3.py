"""A float32 cut into three bfloat16 numbers (csrc/split3.cuh), on the CPU."""
import torch


def parts(x):
    """The parts of float32 numbers, in float64."""
    out = []
    for _ in range(3):
        p = x.to(torch.bfloat16).float()
        out.append(p.double())
        x = x - p
    return out, x


def test_three_parts_are_the_number():
    g = torch.Generator().manual_seed(1)
    x = (1 + torch.rand(1 << 18, generator=g)) * 2.0 ** torch.randint(-110, 60, (1 << 18,), generator=g)
    x[::2] *= -1
    x[:3] = torch.tensor([2.0 ** -110, 2.0 ** -109 - 2.0 ** -133, -(2.0 ** 60)])
    p, rest = parts(x)
    assert torch.equal(sum(p), x.double()) and not rest.any()


def test_what_six_products_leave_out():
    """At most 2^-24 + 2^-34 of the product, reached at 1 + 2^-8 - 2^-17."""
    def left_out(x, w):
        (x0, x1, x2), (w0, w1, w2) = parts(x)[0], parts(w)[0]
        six = x0 * w0 + x0 * w1 + x1 * w0 + x0 * w2 + x1 * w1 + x2 * w0
        return ((x.double() * w.double() - six) / (x.double() * w.double())).abs()
    worst = torch.tensor([1 + 2.0 ** -8 - 2.0 ** -17])
    assert 2.0 ** -24.1 < left_out(worst, worst).item() <= 2.0 ** -24 + 2.0 ** -34
    g = torch.Generator().manual_seed(2)
    x, w = (1 + torch.rand(1 << 20, generator=g) for _ in range(2))
    assert left_out(x, w).max().item() <= 2.0 ** -24 + 2.0 ** -34
