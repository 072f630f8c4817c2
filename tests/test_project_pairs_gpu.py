"""The projection by pairs of CTAs at the k lengths where it begins (576), with ragged rows, columns and k, and a size just past the line (its pairs
would take a round more): against float64."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,d_local,d", [(9408, 576, 704), (9536, 624, 832), (9472, 816, 768), (4736, 640, 4096)])
def test_projection(pkg, torch_cuda, rows, d_local, d):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows + d)
    A = torch.randn(rows, d_local, generator=g, device="cuda").half()
    W = (torch.randn(d_local, d, generator=g, device="cuda") * d_local ** -0.5).half()
    out = torch.full((rows + 1, d), float("nan"), dtype=torch.float16, device="cuda")
    pkg.kernel_status_reset()
    pkg.project(A, W, out, rows, d_local, d)
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0
    want = A.double() @ W.double()
    # fp32 sums of d_local products (exact in fp32), then one rounding to fp16
    bound = want.abs() * 2.0 ** -11 + 2.0 ** -25 + d_local * 2.0 ** -23 * (A.double().abs() @ W.double().abs())
    assert bool(((out[:rows].double() - want).abs() <= bound).all())
    assert torch.isnan(out[rows]).all()


@pytest.mark.parametrize("S,d,H,d_h", [(6464, 592, 8, 64), (4160, 640, 6, 128)])
def test_qkv(pkg, torch_cuda, S, d, H, d_h):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + d)
    X = torch.randn(S, d, generator=g, device="cuda").half()
    W = [(torch.randn(H, d, d_h, generator=g, device="cuda") * d ** -0.5).half() for _ in range(3)]
    out = [torch.full((H, S, d_h), float("nan"), dtype=torch.float16, device="cuda") for _ in range(3)]
    pkg.compute_qkv(X, *W, *out, S, d, H, d_h)
    torch.cuda.synchronize()
    for w, o in zip(W, out):
        want = X.double() @ w.double()
        bound = want.abs() * 2.0 ** -11 + 2.0 ** -25 + d * 2.0 ** -23 * (X.double().abs() @ w.double().abs())
        assert bool(((o.double() - want).abs() <= bound).all())
