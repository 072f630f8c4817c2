"""The merge of split-KV partials against the formula in float64, for the numbers of splits that have a kernel of their own and others, with
empty splits whose O holds no numbers (it is not read) and rows that have only one split."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("split", [2, 3, 4, 5, 6, 8, 15, 16])
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


@pytest.mark.gpu
# Few and many heads, so that all forms of all kernels occur; rows from 64 on: the first 64 rows of a 128-row tile have nothing of a split.
@pytest.mark.parametrize("d_h", [16, 32, 64, 128])
@pytest.mark.parametrize("H,S,split,q_start", [(2, 1152, 3, 64), (80, 1152, 3, 64), (200, 256, 2, 0), (60, 1024, 2, 0)])
@pytest.mark.parametrize("causal", [0, 1])
def test_keys_without_weight_keep_their_values(pkg, torch_cuda, d_h, H, S, split, q_start, causal):
    """All keys of a split score -inf and one of its values is not a number: as without splits, it reaches the rows that have that key (0 * NaN). Rows
    that the mask leaves nothing of that split do not see it."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + d_h)
    q, k, v = (torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))
    first, rows = S // split, S - q_start
    q[..., 0] = q[..., 0].abs() + 0.125
    k[:, first:2 * first, 0] = float("-inf")
    fp = pkg.FlashParams(S, d_h, H, split, causal, d_h ** -0.5)
    ws = [torch.full((n,), float("nan"), device="cuda") for n in (split * rows * H * d_h, split * rows * H, split * rows * H)]
    part = pkg.FlashPartials(*(w.data_ptr() for w in ws), rows)

    def run(v):
        out = torch.full((rows, H, d_h), 7.0, device="cuda")
        pkg.flash_attn_tc_forward(q, k, v, None, part, q_start, rows, fp, o_dtype=pkg.F32)
        pkg.flash_attn_tc_combine(part, out, 0, rows, fp, o_dtype=pkg.F32)
        torch.cuda.synchronize()
        return out
    plain = run(v)
    assert torch.isfinite(plain).all()
    v[:, first, 3] = float("nan")
    out = run(v)
    seen = torch.zeros(rows, H, d_h, dtype=torch.bool, device="cuda")
    seen[first - q_start if causal else 0:, :, 3] = True
    assert torch.equal(torch.isnan(out), seen)
    assert torch.equal(out[~seen], plain[~seen])
