"""The projection kernel behind project() (attn_main.cu:262-273, fp16 data path) against float64 numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,d_local,d", [(64, 16, 64), (128, 64, 64), (128, 128, 1024), (64, 512, 1024),
                                             (256, 1024, 1024), (192, 32, 256), (2048, 512, 512), (4096, 256, 4096),
                                             (128, 4096, 4096), (19072, 128, 1024),
                                             # several tiles per SM, with ragged last rows and columns, one k-block and many
                                             # a block per tile (up to 148 narrow tiles: 64 rows, or d a power of two and
                                             # d_local from 512 on) and just not
                                             (64, 48, 448), (192, 512, 256), (192, 496, 256), (192, 512, 320), (4736, 528, 512), (4800, 528, 512),
                                             (19136, 48, 320), (9536, 16, 704), (4160, 512, 4096), (64, 80, 448)])
def test_projection_matches_float64(pkg, torch_cuda, rows, d_local, d):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows + d_local + d)
    A = torch.randn(rows, d_local, generator=g, device="cuda").to(torch.float16)
    W = (torch.randn(d_local, d, generator=g, device="cuda") / d ** 0.5).to(torch.float16)
    out = torch.full((rows, d), float("nan"), dtype=torch.float16, device="cuda")
    pkg.kernel_status_reset()
    pkg.project(A, W, out, rows, d_local, d)
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0
    ref = A.double() @ W.double()
    err = (out.double() - ref).abs()
    # one fp16 rounding of the result (2^-11 relative) plus fp32 accumulation noise
    bound = ref.abs() * 2 ** -10 + 1e-4 * ref.abs().max()
    assert torch.isfinite(out).all()
    assert bool((err <= bound).all()), float((err - bound).max())


# Ragged last rows and columns, one tile and several per SM, both tile widths; heads that share a tile.
@pytest.mark.parametrize("rows,d_local,d", [(64, 16, 64), (192, 80, 448), (320, 256, 4096), (19136, 48, 320)])
def test_projection_into_mapped_host_memory(pkg, torch_cuda, rows, d_local, d):
    """An output that is not this GPU's own memory gets the same values as one that is."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows + d)
    A = torch.randn(rows, d_local, generator=g, device="cuda").to(torch.float16)
    W = (torch.randn(d_local, d, generator=g, device="cuda") / d ** 0.5).to(torch.float16)
    out = torch.full((rows + 1, d), float("nan"), dtype=torch.float16, device="cuda")
    host = torch.full((rows + 1, d), float("nan"), dtype=torch.float16).pin_memory()
    pkg.kernel_status_reset()
    for o in (out, host):
        pkg.project(A, W, o, rows, d_local, d)
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0
    assert torch.isfinite(out[:rows]).all() and torch.equal(out[:rows].cpu(), host[:rows])
    assert torch.isnan(host[rows]).all()                         # nothing behind the last row
    with pytest.raises(pkg.EfaError, match="16-byte"):
        pkg.project(A, W, host.view(-1)[1:], rows, d_local, d)


@pytest.mark.parametrize("S,d,H_local,d_h", [(192, 80, 3, 64), (4160, 96, 3, 128)])
def test_compute_qkv_into_mapped_host_memory(pkg, torch_cuda, S, d, H_local, d_h):
    """One of the three outputs in host memory is enough for all of them to be written the plain way."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + d)
    X = torch.randn(S, d, generator=g, device="cuda").to(torch.float16)
    W = [torch.randn(H_local, d, d_h, generator=g, device="cuda").to(torch.float16) * 0.1 for _ in range(3)]
    out = [torch.full((H_local, S, d_h), float("nan"), dtype=torch.float16, device="cuda") for _ in range(3)]
    mixed = [out[0].clone(), out[1].cpu().pin_memory(), out[2].clone()]
    for o in (out, mixed):
        pkg.compute_qkv(X, *W, *o, S, d, H_local, d_h)
    torch.cuda.synchronize()
    for a, b in zip(out, mixed):
        assert torch.isfinite(a).all() and torch.equal(a.cpu(), b.cpu())


def test_projection_rejects_bad_shapes(pkg, torch_cuda):
    torch = torch_cuda
    A = torch.zeros(128, 64, dtype=torch.float16, device="cuda")
    W = torch.zeros(64, 64, dtype=torch.float16, device="cuda")
    out = torch.zeros(128, 64, dtype=torch.float16, device="cuda")
    with pytest.raises(pkg.EfaError):
        pkg.project(A, W, out, 100, 64, 64)
    with pytest.raises(pkg.EfaError):
        pkg.project(A, W, out, 128, 24, 64)
    with pytest.raises(pkg.EfaError):
        pkg.project(A, W, out, 128, 64, 96)


def test_a_launch_that_is_refused_leaves_no_error_behind(pkg, torch_cuda):
    """More row tiles than a grid has (65535): the call fails, and the next one does not inherit the error."""
    torch = torch_cuda
    rows = 65536 * 128
    A = torch.zeros(rows, 16, dtype=torch.float16, device="cuda")
    W = torch.zeros(16, 64, dtype=torch.float16, device="cuda")
    out = torch.zeros(rows, 64, dtype=torch.float16, device="cuda")
    with pytest.raises(pkg.EfaError, match="proj_gemm_kernel"):
        pkg.project(A, W, out, rows, 16, 64)
    x = torch.arange(64, dtype=torch.float32, device="cuda")
    y = torch.empty(64, dtype=torch.float16, device="cuda")
    pkg.convert_f32_to_f16(x, y, 64)
    assert torch.equal(y, x.half())
    pkg.project(A, W, out, 128, 16, 64)
    torch.cuda.synchronize()


@pytest.mark.parametrize("S,d,H_local,d_h", [(512, 512, 4, 128), (1024, 1024, 2, 64), (2048, 256, 4, 64),
                                            # tiles that span heads and tensors, ragged rows, columns and k; several tiles per SM
                                            (192, 80, 3, 64), (64, 16, 1, 64), (320, 144, 1, 128), (8256, 208, 5, 64), (4160, 96, 3, 128)])
def test_compute_qkv_matches_float64(pkg, torch_cuda, S, d, H_local, d_h):
    """The step before the block (compute_qkv, attn_main.cu:127-153) on fp16 data, head-major output."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + d)
    X = (torch.rand(S, d, generator=g, device="cuda") * 2 - 1).to(torch.float16)
    W = [((torch.rand(H_local, d, d_h, generator=g, device="cuda") * 2 - 1) * 0.15).to(torch.float16) for _ in range(3)]
    out = [torch.full((H_local, S, d_h), float("nan"), dtype=torch.float16, device="cuda") for _ in range(3)]
    pkg.compute_qkv(X, W[0], W[1], W[2], out[0], out[1], out[2], S, d, H_local, d_h)
    torch.cuda.synchronize()
    for t in range(3):
        ref = torch.einsum("sk,hkj->hsj", X.double(), W[t].double())
        err = (out[t].double() - ref).abs()
        assert torch.isfinite(out[t]).all()
        assert bool((err <= ref.abs() * 2 ** -10 + 1e-4 * ref.abs().max()).all())
    with pytest.raises(pkg.EfaError, match="d_h"):
        pkg.compute_qkv(X, W[0], W[1], W[2], out[0], out[1], out[2], S, d, H_local, 32)


# Pairs of CTAs to a tile (see in_pairs): one row past a tile's first half, ragged rows, columns and k; fewer tiles than pairs of SMs
# and several per pair; just below the limits.
@pytest.mark.parametrize("rows,d_local,d", [(256, 2048, 4096), (320, 2064, 8192), (2048, 2048, 2048), (9408, 832, 640), (9536, 848, 704),
                                            (9408, 816, 640), (4160, 4080, 1088), (19136, 1040, 576)])
def test_projection_by_pairs_matches_float64(pkg, torch_cuda, rows, d_local, d):
    test_projection_matches_float64(pkg, torch_cuda, rows, d_local, d)


@pytest.mark.parametrize("S,d,H_local,d_h", [(6464, 848, 8, 64), (8256, 1040, 5, 64), (1088, 2064, 16, 128), (4160, 2048, 3, 128)])
def test_compute_qkv_by_pairs_matches_float64(pkg, torch_cuda, S, d, H_local, d_h):
    """Tiles whose two CTAs take columns of different heads and tensors."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + d)
    X = torch.randn(S, d, generator=g, device="cuda").to(torch.float16)
    W = [(torch.randn(H_local, d, d_h, generator=g, device="cuda") * d ** -0.5).to(torch.float16) for _ in range(3)]
    out = [torch.full((H_local, S, d_h), float("nan"), dtype=torch.float16, device="cuda") for _ in range(3)]
    pkg.kernel_status_reset()
    for _ in range(3):
        pkg.compute_qkv(X, W[0], W[1], W[2], out[0], out[1], out[2], S, d, H_local, d_h)
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0
    for t in range(3):
        ref = torch.einsum("sk,hkj->hsj", X.double(), W[t].double())
        err = (out[t].double() - ref).abs()
        assert torch.isfinite(out[t]).all()
        assert bool((err <= ref.abs() * 2 ** -10 + 1e-4 * ref.abs().max()).all())


@pytest.mark.parametrize("S,H,d_h", [(4096, 16, 128), (20480, 14, 64)])
def test_fp32_projection_by_pairs(pkg, torch_cuda, S, H, d_h):
    """fp32 sums of the block's projection: the fp16 result is their rounding."""
    torch = torch_cuda
    d = H * d_h
    p = pkg.make_params(S, d, H, 64)
    g = torch.Generator(device="cuda").manual_seed(S)
    dev = [torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3)]
    dev.append(torch.randn(d, d, generator=g, device="cuda", dtype=torch.float16) * d ** -0.5)
    w = pkg.Weights(*(t.data_ptr() for t in dev))
    ctx = pkg.make_ctx(pkg.World(), ncomm=1)
    try:
        half = torch.full((S, d), float("nan"), dtype=torch.float16, device="cuda")
        full = torch.full((S, d), float("nan"), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        pkg.run_mode(ctx, pkg.MODE_MEGATRON, w, half, p)
        p.proj_f32 = 1
        pkg.run_mode(ctx, pkg.MODE_MEGATRON, w, full, p)
    finally:
        pkg.destroy_ctx(ctx)
    assert torch.isfinite(full).all() and torch.equal(full.to(torch.float16), half)


# A cluster per tile (see k_parts): eight, four and two parts of k, also of unequal length and with a ragged last k-block; ragged rows
# and columns; at the limits of each and just past them.
@pytest.mark.parametrize("rows,d_local,d", [(64, 4080, 64), (128, 2048, 1024), (128, 2032, 1088), (192, 1040, 448), (2048, 1024, 256), (2112, 1024, 256),
                                            (320, 976, 704), (320, 960, 704), (4096, 2560, 256), (4160, 2560, 256), (1984, 2512, 448), (1984, 2480, 448)])
def test_projection_by_parts_of_k_matches_float64(pkg, torch_cuda, rows, d_local, d):
    for _ in range(3):
        test_projection_matches_float64(pkg, torch_cuda, rows, d_local, d)


@pytest.mark.parametrize("S,d,H_local,d_h", [(1024, 3008, 1, 64), (192, 1040, 3, 64), (64, 2064, 2, 128)])
def test_compute_qkv_by_parts_of_k_matches_float64(pkg, torch_cuda, S, d, H_local, d_h):
    test_compute_qkv_by_pairs_matches_float64(pkg, torch_cuda, S, d, H_local, d_h)


def test_projection_by_parts_of_k_into_mapped_host_memory(pkg, torch_cuda):
    test_projection_into_mapped_host_memory(pkg, torch_cuda, 192, 1040, 448)


@pytest.mark.parametrize("S,d,H_local,d_h", [(192, 1040, 3, 64), (1024, 3008, 1, 64), (64, 2064, 2, 128)])
def test_compute_qkv_by_parts_of_k_into_mapped_host_memory(pkg, torch_cuda, S, d, H_local, d_h):
    """Where k is summed in parts it is so for any output memory: the same bits. Nothing is written past the last row, and an output that
    is not 16-byte aligned is refused."""
    torch = torch_cuda
    test_compute_qkv_into_mapped_host_memory(pkg, torch, S, d, H_local, d_h)
    X = torch.ones(S, d, dtype=torch.float16, device="cuda")
    W = [torch.ones(H_local, d, d_h, dtype=torch.float16, device="cuda") for _ in range(3)]
    host = [torch.full((H_local * S * d_h + 64,), float("nan"), dtype=torch.float16).pin_memory() for _ in range(3)]
    pkg.compute_qkv(X, *W, *host, S, d, H_local, d_h)
    torch.cuda.synchronize()
    for o in host:
        assert bool((o[:-64] == d).all()) and torch.isnan(o[-64:]).all()
    with pytest.raises(pkg.EfaError, match="16-byte"):
        pkg.compute_qkv(X, *W, host[0], host[1].view(-1)[1:], host[2], S, d, H_local, d_h)


# Eight, four and two parts of k.
@pytest.mark.parametrize("rows,d_local,d", [(64, 4080, 64), (192, 1040, 448), (1984, 2512, 448)])
def test_parts_of_k_give_the_same_bits_every_time(pkg, torch_cuda, rows, d_local, d):
    """Whatever the stream and whatever runs beside, a call of the same sizes adds the parts in the same order."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows)
    A = torch.randn(rows, d_local, generator=g, device="cuda").to(torch.float16)
    W = (torch.randn(d_local, d, generator=g, device="cuda") / d ** 0.5).to(torch.float16)
    outs = [torch.full((rows, d), float("nan"), dtype=torch.float16, device="cuda") for _ in range(8)]
    streams = [torch.cuda.Stream(priority=-(i & 1)) for i in range(4)]
    big = torch.randn(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        with torch.cuda.stream(streams[(i + 1) % 4]):
            torch.mm(big, big)
        pkg.project(A, W, out, rows, d_local, d, streams[i % 4])
    torch.cuda.synchronize()
    assert torch.isfinite(outs[0]).all() and all(torch.equal(o, outs[0]) for o in outs)
