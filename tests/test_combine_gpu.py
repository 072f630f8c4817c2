"""The merge of split-KV partials against the formula in float64, for the numbers of splits that have a kernel of their own and others, with
empty splits whose O holds no numbers (it is not read) and rows that have only one split."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("split", [2, 3, 4, 8, 16])
@pytest.mark.parametrize("rows,row0,H,d_h,f16", [(64, 0, 3, 16, True), (192, 64, 5, 64, False), (2048, 0, 2, 128, True)])
def test_merge(pkg, torch_cuda, split, rows, row0, H, d_h, f16):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(split + rows)
    n = row0 + rows + 64
    O = torch.randn(split, n, H, d_h, generator=g, device="cuda")
    m = torch.randn(split, n, H, generator=g, device="cuda") * 20
    l = torch.rand(split, n, H, generator=g, device="cuda") * 50 + 1
    empty = torch.rand(split, n, H, generator=g, device="cuda") < 0.4
    keep = torch.randint(0, split, (n, H), generator=g, device="cuda")
    empty.scatter_(0, keep[None], False)
    m[empty], l[empty] = float("-inf"), 0.0
    O[empty] = 0.0
    part = pkg.FlashPartials(O.data_ptr(), m.data_ptr(), l.data_ptr(), n)
    S = 64 * split * 64
    fp = pkg.FlashParams(S, d_h, H, split, 1, 1.0)
    w = torch.exp2(m.double() - m.double().max(0).values)
    want = ((w[..., None] * O.double()).sum(0) / (w * l.double()).sum(0)[..., None])[row0:row0 + rows].reshape(rows, H * d_h)
    size = ((w[..., None] * O.double().abs()).sum(0) / (w * l.double()).sum(0)[..., None])[row0:row0 + rows].reshape(rows, H * d_h)
    for poison in (False, True):
        if poison:
            O[empty] = float("nan")
        out = torch.full((rows, H * d_h), float("nan"), device="cuda", dtype=torch.float16 if f16 else torch.float32)
        pkg.flash_attn_tc_combine(part, out, row0, rows, fp, o_dtype=pkg.F16 if f16 else pkg.F32)
        torch.cuda.synchronize()
        # fp32: 2^-22 for each exponential, 2^-24 for each of split sums and three more roundings; then the result's own
        bound = size * (2 * 2.0 ** -22 + (split + 4) * 2.0 ** -23) + (want.abs() * 2.0 ** -11 + 2.0 ** -25 if f16 else 0)
        assert bool(((out.double() - want).abs() <= bound).all())
