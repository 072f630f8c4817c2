"""Kernels whose blocks start before the kernel ahead of them in the stream has ended: a chain of calls in which every one
reads what the one before it wrote gives the same bits as the same chain with a synchronisation after every call."""
import pytest

pytestmark = pytest.mark.gpu


# One wave and several of every kernel; split keys with their merge; a short last wave in a launch of its own (13 heads of 128);
# items of four chains; the kernel of small heads and few keys.
@pytest.mark.parametrize("S,H,d_h,split", [(192, 2, 64, 1), (1024, 4, 64, 4), (4096, 13, 128, 1), (2048, 16, 128, 2), (512, 40, 32, 1), (256, 80, 32, 1)])
@pytest.mark.parametrize("side", [False, True], ids=["default stream", "other stream"])
def test_a_chain_of_calls_needs_no_synchronisation(pkg, torch_cuda, S, H, d_h, split, side):
    torch = torch_cuda
    d = H * d_h
    p = pkg.make_params(S, d, H, 64, 2, split, 1 if d_h == 64 else 0)
    g = torch.Generator(device="cuda").manual_seed(S + H)
    X = [torch.randn(S, d, generator=g, device="cuda", dtype=torch.float16) for _ in range(3)]
    W = [torch.randn(d, d, generator=g, device="cuda", dtype=torch.float16) * d ** -0.5 for _ in range(2)]
    qkv = [torch.empty(H, S, d_h, device="cuda", dtype=torch.float16) for _ in range(3)]
    O, T, Y = (torch.empty(S, d, device="cuda", dtype=torch.float16) for _ in range(3))
    ws = [torch.empty(n, device="cuda") for n in (split * S * d, split * S * H, split * S * H)]
    part = pkg.FlashPartials(*(w.data_ptr() for w in ws), S) if split > 1 else None
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()

    def chain(x, sync):
        after = torch.cuda.synchronize if sync else (lambda: None)
        for k in range(3):                                   # the tensors of one pass are overwritten by the next
            pkg.project(x, W[k & 1], T, S, d, d, stream)
            after()
            for t in range(3):
                qkv[t].copy_(T.view(S, H, d_h).transpose(0, 1))
                T.mul_(0.5)
            after()
            pkg.flash_attn_tc_forward(*qkv, O, part, 0, S, p.flash_tc, stream)
            after()
            if part is not None:
                pkg.flash_attn_tc_combine(part, O, 0, S, p.flash_tc, stream)
                after()
            pkg.project(O, W[0], T, S, d, d, stream)
            after()
            pkg.project(T, W[1], Y, S, d, d, stream)
            after()
            x = Y
        return Y.clone()

    torch.cuda.synchronize()
    pkg.kernel_status_reset()
    with torch.cuda.stream(stream):
        want = [chain(x, True) for x in X]
        got = [chain(x, False) for x in X for _ in range(2)]
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0
    for i, y in enumerate(got):
        assert torch.isfinite(y).all() and torch.equal(y, want[i // 2])


@pytest.mark.parametrize("S,H,d_h,split", [(192, 2, 64, 1), (1024, 4, 64, 4), (4096, 13, 128, 1), (512, 40, 32, 1), (256, 80, 32, 1)])
def test_a_captured_chain_with_joins_keeps_its_order(pkg, torch_cuda, S, H, d_h, split):
    """The same kernels in a CUDA graph, where a call also follows work of another stream (a join), on inputs that change from replay to
    replay: as the calls give one by one."""
    torch = torch_cuda
    d = H * d_h
    p = pkg.make_params(S, d, H, 64, 2, split, 0)
    g = torch.Generator(device="cuda").manual_seed(S + H)
    X = [torch.randn(S, d, generator=g, device="cuda", dtype=torch.float16) for _ in range(3)]
    W = [torch.randn(d, d, generator=g, device="cuda", dtype=torch.float16) * d ** -0.5 for _ in range(2)]
    x, half, T, U, O, Y = (torch.zeros(S, d, device="cuda", dtype=torch.float16) for _ in range(6))
    qkv = [torch.zeros(H, S, d_h, device="cuda", dtype=torch.float16) for _ in range(3)]
    ws = [torch.zeros(n, device="cuda") for n in (split * S * d, split * S * H, split * S * H)]
    part = pkg.FlashPartials(*(w.data_ptr() for w in ws), S) if split > 1 else None
    side = torch.cuda.Stream()

    def chain(sync):
        after = torch.cuda.synchronize if sync else (lambda: None)
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        pkg.project(x, W[0], T, S, d, d, main)
        after()
        with torch.cuda.stream(side):                        # beside the first projection
            torch.mul(x, 0.5, out=half)
            pkg.project(half, W[1], U, S, d, d, side)
        after()
        main.wait_stream(side)                               # the next call follows both
        pkg.project(U, W[0], Y, S, d, d, main)
        after()
        for t, src in enumerate((T, U, Y)):
            qkv[t].copy_(src.view(S, H, d_h).transpose(0, 1))
        after()
        pkg.flash_attn_tc_forward(*qkv, O, part, 0, S, p.flash_tc, main)
        after()
        if part is not None:
            pkg.flash_attn_tc_combine(part, O, 0, S, p.flash_tc, main)
            after()
        pkg.project(O, W[1], Y, S, d, d, main)
        after()

    want = []
    for v in X:
        x.copy_(v)
        chain(True)
        want.append(Y.clone())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(False)
    pkg.kernel_status_reset()
    for i in (0, 1, 2, 1, 0):
        x.copy_(X[i])
        graph.replay()
        assert torch.isfinite(Y).all() and torch.equal(Y, want[i])
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0
