"""The exact float form's square root and arctangent (sqrt_lv, atan2_lv in csrc/frac_kernels.cuh), one value at a time and as
packed pairs: the root is the correctly rounded one for every float, the arctangent no worse than CUDA's."""

import pytest

pytestmark = pytest.mark.gpu


def probe(ag, disp, a, b):
    import torch
    out = [torch.empty_like(a) for _ in range(4)]
    torch.cuda.synchronize()
    assert ag.library().agwn_probe_math_f32(disp.handle, a.data_ptr(), b.data_ptr(), a.numel(),
                                            *(o.data_ptr() for o in out)) == 0
    return out


def same(a, b):
    import torch
    return bool((torch.eq(a.view(torch.int32), b.view(torch.int32)) | (torch.isnan(a) & torch.isnan(b))).all())


def test_root_of_every_float():
    """All 2^32 of them, zeros, subnormals, infinities, NaN and negative ones included: the approximate reciprocal root that
    the chip returns decides whether one correction is enough, so none is left out."""
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    with ag.CudaDispatcher() as disp:
        step = 1 << 26
        for first in range(-(1 << 31), 1 << 31, step):
            a = torch.arange(first, first + step, dtype=torch.int64, device="cuda").to(torch.int32).view(torch.float32)
            root, root2, _, _ = probe(ag, disp, a, a)
            # a double's root rounded to float is the float's (the double has more than twice its digits)
            want = a.double().sqrt().float()
            assert same(root, want) and same(root2, want)


def arguments(kind, n=1 << 22):
    import torch
    g = torch.Generator(device="cuda").manual_seed(len(kind))
    u = lambda lo, hi: torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo  # noqa: E731
    if kind == "normal":
        y, x = (torch.randn(n, generator=g, device="cuda", dtype=torch.float64) for _ in range(2))
    elif kind == "small angles":
        y, x = u(0.0, 0.05), u(1.0, 2.0)
    elif kind == "near the diagonals":
        y = u(1.0, 2.0)
        x = y * u(0.999, 1.001) * torch.where(u(0, 1) < 0.5, 1.0, -1.0)
    else:  # "skewed": ratios of any size, all quadrants, scales up to 2^+-90
        s = torch.exp2(u(-60.0, 60.0))
        y = s * torch.exp2(u(-30.0, 30.0)) * torch.where(u(0, 1) < 0.5, 1.0, -1.0)
        x = s * torch.where(u(0, 1) < 0.5, 1.0, -1.0)
    return y.float(), x.float()


@pytest.mark.parametrize("kind", ["normal", "small angles", "near the diagonals", "skewed"])
def test_arctangent_no_worse_than_cuda(kind):
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    y, x = arguments(kind)
    with ag.CudaDispatcher() as disp:
        _, _, angle, angle2 = probe(ag, disp, y, x)
    assert same(angle, angle2)
    want = torch.atan2(y.double(), x.double())
    w = want.float()
    ulp = (torch.nextafter(w.abs(), torch.full_like(w, float("inf"))).double() - w.abs().double())

    def errors(a):
        e = (a.double() - want).abs() / ulp
        return float(e.mean()), float(e.max())
    ours, cuda = errors(angle), errors(torch.atan2(y, x))
    assert ours[0] <= cuda[0] and ours[1] <= cuda[1], (ours, cuda)


def test_arctangent_of_special_values():
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    v = torch.tensor([0.0, -0.0, 1.0, -1.0, float("inf"), -float("inf"), float("nan"), 1e-45, -1e-45, 1.2e-38, 3.4e38, -3.4e38,
                      2.0 ** 100, 2.0 ** -100, 2.0 ** -101], device="cuda")
    y, x = (t.reshape(-1).contiguous() for t in torch.meshgrid(v, v, indexing="ij"))
    with ag.CudaDispatcher() as disp:
        _, _, angle, angle2 = probe(ag, disp, y, x)
    want = torch.atan2(y.double(), x.double())
    assert same(angle, angle2) and torch.equal(torch.isnan(angle), torch.isnan(want))
    ok = ~torch.isnan(angle)
    assert torch.equal(torch.signbit(angle[ok]), torch.signbit(want[ok]))
    w = want[ok].float()
    ulp = torch.nextafter(w.abs(), torch.full_like(w, float("inf"))).double() - w.abs().double()
    assert float(((angle[ok].double() - want[ok]).abs() / ulp).max()) <= 2.0
