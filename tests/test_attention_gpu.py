"""The attention kernel behind flash_attn_tc_forward against the CPU full-softmax checker, on the
reference's own test shapes (attn_tests.cu:70-85) and on the edge cases of the launch interface."""
import numpy as np
import pytest

from conftest import REFERENCE_CASES, REFERENCE_SEEDS
from helpers import assert_close, ref_inputs_f16, to_dev

pytestmark = pytest.mark.gpu


def run_attention(pkg, torch, p, dev, q_start, q_rows, o_dtype, tile_rows=None, poison=True):
    """One launch over rows [q_start, q_start + q_rows), split partials combined; returns (O, counters)."""
    Qd, Kd, Vd = dev[:3]
    tdtype = torch.float16 if o_dtype == pkg.F16 else torch.float32
    O = torch.full((q_rows, p.d_local), float("nan") if poison else 0.0, dtype=tdtype, device="cuda")
    part = None
    keep = []
    if p.split > 1:
        Op = torch.full((p.split, q_rows, p.d_local), float("nan"), dtype=torch.float32, device="cuda")
        mp = torch.full((p.split, q_rows, p.H_local), float("nan"), dtype=torch.float32, device="cuda")
        lp = torch.full((p.split, q_rows, p.H_local), float("nan"), dtype=torch.float32, device="cuda")
        keep = [Op, mp, lp]
        part = pkg.FlashPartials(Op.data_ptr(), mp.data_ptr(), lp.data_ptr(), q_rows)
    counters = None
    if tile_rows:
        counters = torch.zeros((q_rows + tile_rows - 1) // tile_rows, dtype=torch.int32, device="cuda")
    pkg.kernel_status_reset()
    pkg.flash_attn_tc_forward(Qd, Kd, Vd, O, part, q_start, q_rows, p.flash_tc, None, counters, tile_rows or 0, o_dtype)
    if p.split > 1:
        pkg.flash_attn_tc_combine(part, O, 0, q_rows, p.flash_tc, None, o_dtype)
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0, f"kernel status {pkg.kernel_status()}"
    return O, counters


@pytest.mark.parametrize("case", REFERENCE_CASES, ids=lambda c: "S%d_d%d_H%d_t%d_n%d_s%d_c%d" % c)
def test_reference_shapes(pkg, oracle, torch_cuda, case):
    torch = torch_cuda
    S, d, H, tile, nbuf, split, causal = case
    p = pkg.make_params(S, d, H, tile, nbuf, split, causal)
    seeds = REFERENCE_SEEDS if S <= 1024 else REFERENCE_SEEDS[:1]
    for seed in seeds:
        bits, vals = ref_inputs_f16(oracle, S, d, H, 1, 0, seed)
        ref = oracle.attention_rows(vals[0], vals[1], vals[2], causal)
        dev = to_dev(torch, bits)
        for o_dtype in (pkg.F16, pkg.F32):
            O, counters = run_attention(pkg, torch, p, dev, 0, S, o_dtype, tile_rows=tile)
            assert_close(oracle, O.float().cpu().numpy(), ref, f"seed {seed} dtype {o_dtype}")
            assert counters.cpu().tolist() == [pkg.blocks_per_tile(p)] * (S // tile)


@pytest.mark.parametrize("S,d,H,causal,split", [(192, 256, 4, 0, 1), (192, 256, 4, 1, 1), (320, 128, 2, 1, 1),
                                               (192, 64, 4, 1, 3), (448, 512, 4, 0, 1)])
def test_sequence_lengths_that_are_odd_multiples_of_64(pkg, oracle, torch_cuda, S, d, H, causal, split):
    torch = torch_cuda
    p = pkg.make_params(S, d, H, 64, 2, split, causal)
    assert pkg.attn_check_params(p) is None
    bits, vals = ref_inputs_f16(oracle, S, d, H, 1, 0, 42)
    ref = oracle.attention_rows(vals[0], vals[1], vals[2], causal)
    O, counters = run_attention(pkg, torch, p, to_dev(torch, bits), 0, S, pkg.F32, tile_rows=64)
    assert_close(oracle, O.cpu().numpy(), ref)
    assert counters.cpu().tolist() == [pkg.blocks_per_tile(p)] * (S // 64)


@pytest.mark.parametrize("q_start,q_rows,tile_rows", [(0, 64, 64), (64, 64, 64), (128, 192, 64), (256, 256, 128), (448, 64, 64), (192, 320, 64)])
@pytest.mark.parametrize("causal", [0, 1])
def test_row_windows(pkg, oracle, torch_cuda, q_start, q_rows, tile_rows, causal):
    """Launches over a window of rows: O and the counters are indexed from the launch's first row,
    keys and the causal mask from the absolute row (flash_attn_tc.cuh:39-44)."""
    torch = torch_cuda
    S, d, H = 512, 256, 4
    p = pkg.make_params(S, d, H, tile_rows, 2, 1, causal)
    bits, vals = ref_inputs_f16(oracle, S, d, H, 1, 0, 123)
    rows = np.arange(q_start, q_start + q_rows, dtype=np.int32)
    ref = oracle.attention_rows(vals[0], vals[1], vals[2], causal, rows)
    O, counters = run_attention(pkg, torch, p, to_dev(torch, bits), q_start, q_rows, pkg.F16, tile_rows=tile_rows)
    assert_close(oracle, O.float().cpu().numpy(), ref)
    total = sum(counters.cpu().tolist())
    assert total == (q_rows // 64) * p.H_local


def test_split_partials_follow_the_reference_layout(pkg, oracle, torch_cuda):
    """m_part is the row max of scale*log2(e)*s, l_part the denominator, O_part unnormalised
    (flash_attn_tc.cuh:25-34): recombining them on the host must give the checker's rows."""
    torch = torch_cuda
    S, d, H, split = 512, 256, 4, 4
    p = pkg.make_params(S, d, H, 128, 2, split, 0)
    bits, vals = ref_inputs_f16(oracle, S, d, H, 1, 0, 777)
    dev = to_dev(torch, bits)
    Op = torch.zeros((split, S, p.d_local), dtype=torch.float32, device="cuda")
    mp = torch.zeros((split, S, p.H_local), dtype=torch.float32, device="cuda")
    lp = torch.zeros((split, S, p.H_local), dtype=torch.float32, device="cuda")
    part = pkg.FlashPartials(Op.data_ptr(), mp.data_ptr(), lp.data_ptr(), S)
    pkg.flash_attn_tc_forward(dev[0], dev[1], dev[2], None, part, 0, S, p.flash_tc, None, None, 0, pkg.F32)
    torch.cuda.synchronize()
    O_part, m, l = Op.cpu().numpy().astype(np.float64), mp.cpu().numpy().astype(np.float64), lp.cpu().numpy().astype(np.float64)
    M = m.max(axis=0)
    w = np.exp2(m - M)                                   # [split][S][H]
    L = (w * l).sum(axis=0)
    wfull = np.repeat(w, p.d_h, axis=2)
    O = (wfull * O_part).sum(axis=0) / np.repeat(L, p.d_h, axis=1)
    ref = oracle.attention_rows(vals[0], vals[1], vals[2], 0)
    assert_close(oracle, O.astype(np.float32), ref)
    # the per-split maxima are those of the scaled scores of that key range, in the log2 domain
    s = (vals[0][0, 5].astype(np.float64) @ vals[1][0, :128].astype(np.float64).T) * p.flash_tc.scale * 1.4426950408889634
    assert abs(m[0, 5, 0] - s.max()) < 1e-3


def test_illegal_launches_are_rejected(pkg, torch_cuda):
    torch = torch_cuda
    p = pkg.make_params(256, 256, 4, 64)
    x = torch.zeros(4 * 256 * 64, dtype=torch.float16, device="cuda")
    O = torch.zeros(256 * 256, dtype=torch.float16, device="cuda")
    with pytest.raises(pkg.EfaError, match="multiple of 64"):
        pkg.flash_attn_tc_forward(x, x, x, O, None, 0, 96, p.flash_tc)
    with pytest.raises(pkg.EfaError, match="outside"):
        pkg.flash_attn_tc_forward(x, x, x, O, None, 192, 128, p.flash_tc)
    bad = pkg.make_params(256, 192, 4, 64).flash_tc
    with pytest.raises(pkg.EfaError, match="d_h"):
        pkg.flash_attn_tc_forward(x, x, x, O, None, 0, 64, bad)
    p2 = pkg.make_params(256, 256, 4, 64, split=2)
    with pytest.raises(pkg.EfaError, match="workspace"):
        pkg.flash_attn_tc_forward(x, x, x, O, None, 0, 64, p2.flash_tc)


def test_convert_f32_to_f16(pkg, torch_cuda):
    torch = torch_cuda
    x = torch.randn(100003, device="cuda", dtype=torch.float32) * 3
    y = torch.zeros(100003, device="cuda", dtype=torch.float16)
    pkg.convert_f32_to_f16(x, y, x.numel())
    torch.cuda.synchronize()
    assert torch.equal(y, x.to(torch.float16))


@pytest.mark.parametrize("S,H_local,d_h,causal", [(16384, 2, 64, 0), (32768, 2, 64, 1), (65536, 2, 64, 1), (65536, 2, 64, 0), (32768, 4, 128, 1)],
                         ids=lambda v: str(v))
def test_full_size_rank_shards_on_sampled_rows(pkg, oracle, torch_cuda, S, H_local, d_h, causal):
    """One rank's shard of the eight-GPU configurations of the benchmark plan (two heads of d_h = 64 at
    S = 16k/32k/64k; four heads of d_h = 128 at S = 32k), N(0,1) inputs, checked on rows from the first, last
    and interior tiles, plus a size-independent property: with V = 1 every output element is exactly 1."""
    torch = torch_cuda
    R = 8
    p = pkg.make_params(S, R * H_local * d_h, R * H_local, 128, 2, 1, causal, R)
    assert p.H_local == H_local
    bits = [np.zeros((H_local, S, d_h), np.uint16) for _ in range(3)] + [np.zeros((p.d_local, p.d), np.uint16)]
    pkg.fill_host_inputs(p, 3, 42, pkg.RECIPE_NORMAL, *bits)
    vals = [oracle.widen_f16(b) for b in bits[:3]]
    rng = np.random.default_rng(S + d_h)
    rows = np.unique(np.concatenate([np.arange(0, 24), np.arange(S - 24, S), rng.integers(24, S - 24, 48)])).astype(np.int32)
    ref = oracle.attention_rows(vals[0], vals[1], vals[2], causal, rows)
    dev = to_dev(torch, bits[:3])
    O, counters = run_attention(pkg, torch, p, dev, 0, S, pkg.F16, tile_rows=128)
    assert counters.cpu().tolist() == [pkg.blocks_per_tile(p)] * (S // 128)
    assert_close(oracle, O[torch.from_numpy(rows.astype(np.int64)).cuda()].float().cpu().numpy(), ref)
    ones = torch.ones((H_local, S, d_h), dtype=torch.float16, device="cuda")
    O1, _ = run_attention(pkg, torch, p, [dev[0], dev[1], ones], 0, S, pkg.F32)
    assert float((O1 - 1.0).abs().max()) < 2e-3


def check_against_float64(pkg, torch, H, d_h, S, q_start, q_rows, split, causal, growing=True, tile_rows=64):
    """One launch against float64; growing: on rows whose maximum keeps growing along the keys, so that the exponent
    offset moves after the first stages too."""
    p = pkg.make_params(S, H * d_h, H, 64, 2, split, causal)
    g = torch.Generator(device="cuda").manual_seed(S + d_h + H)
    dev = [torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3)]
    if growing:
        dev[1] *= torch.linspace(0.5, 6.0, S, device="cuda", dtype=torch.float16)[None, :, None]
    O, counters = run_attention(pkg, torch, p, dev, q_start, q_rows, pkg.F32, tile_rows=tile_rows)
    assert torch.isfinite(O).all()
    if tile_rows:
        assert counters.cpu().tolist() == [H * split * tile_rows // 64] * (q_rows // tile_rows)
    rows = torch.arange(q_start, q_start + q_rows, device="cuda")[:, None]
    for h in range(H):
        q, k, v = (t[h].double() for t in dev)
        s = q[q_start:q_start + q_rows] @ k.T * p.flash_tc.scale
        if causal:
            s = s.masked_fill(torch.arange(S, device="cuda")[None, :] > rows, float("-inf"))
        w = torch.softmax(s, dim=-1)
        ref = w @ v
        # Every softmax weight is rounded to fp16 (2^-11 of it) or, below 2^-14 of the largest, to a multiple of 2^-25; the
        # offset may lag the maximum by 2^8. fp32 scores of up to about 100 carry 1e-5 of relative error into the weights.
        bound = (w * 2 ** -11 + 2.0 ** -24) @ v.abs() + 1e-4 * ref.abs().max()
        err = (O[:, h * d_h:(h + 1) * d_h].double() - ref).abs()
        assert bool((err <= bound).all()), (h, float((err - bound).max()))


def form(pkg, H, d_h, S, q_start, q_rows, split, causal):
    """The kernel forms that a launch takes: "256", "128", both behind one another, or "tiles"."""
    plan = pkg.flash_attn_tc_plan(pkg.make_params(S, H * d_h, H, 64, 2, split, causal).flash_tc, q_start, q_rows)
    return "+".join(n for n, items in (("256", plan.items_256), ("128", plan.items_128), ("tiles", plan.tiles)) if items)


# One to seven key stages (more than the ring of two keeps), ragged last blocks, rows that see no key of a split, both directions of the mask.
@pytest.mark.parametrize("d_h", [16, 32])
@pytest.mark.parametrize("H,S,q_start,q_rows,split,causal", [
    (160, 64, 0, 64, 1, 0), (100, 256, 0, 256, 1, 1), (152, 192, 64, 128, 1, 1), (80, 640, 320, 320, 1, 0), (50, 640, 0, 640, 1, 0),
    (80, 448, 0, 192, 1, 1), (12, 1024, 0, 1024, 4, 1), (25, 1280, 192, 576, 2, 0), (160, 384, 0, 384, 1, 0), (160, 448, 192, 256, 1, 0), (75, 640, 0, 640, 1, 1),
    (75, 896, 0, 896, 1, 1), (90, 640, 320, 320, 1, 1), (190, 640, 512, 128, 1, 1)])
def test_single_tiles_against_float64(pkg, torch_cuda, d_h, H, S, q_start, q_rows, split, causal):
    assert form(pkg, H, d_h, S, q_start, q_rows, split, causal) == "tiles"
    check_against_float64(pkg, torch_cuda, H, d_h, S, q_start, q_rows, split, causal)


# As few keys that go as items of the four chains.
@pytest.mark.parametrize("d_h", [16, 32])
@pytest.mark.parametrize("H,S,q_start,q_rows,split,causal,want", [
    (60, 640, 320, 320, 1, 0, "256"), (40, 640, 0, 640, 1, 0, "256"), (16, 1280, 192, 576, 2, 0, "256"), (10, 2048, 0, 2048, 1, 1, "128"),
    (148, 512, 0, 512, 1, 0, "256"), (32, 1024, 0, 1024, 1, 1, "128")])
def test_few_keys_as_items_against_float64(pkg, torch_cuda, d_h, H, S, q_start, q_rows, split, causal, want):
    assert form(pkg, H, d_h, S, q_start, q_rows, split, causal) == want
    check_against_float64(pkg, torch_cuda, H, d_h, S, q_start, q_rows, split, causal)


# Key stages per 128-row block at which the two softmax warpgroups of a 128-row item get none, one, an odd and an even
# number: three heads take that form. Forty heads take it where they are at most 148 such items (the shapes of one split, and
# 64 rows), else single tiles (d_h 16 and 32) or 256-row items (d_h 64 and 128).
@pytest.mark.parametrize("H", [3, 40])
@pytest.mark.parametrize("d_h", [16, 32, 64, 128])
@pytest.mark.parametrize("S,q_start,q_rows,split,causal", [
    (64, 0, 64, 1, 0), (128, 0, 128, 1, 1), (192, 64, 128, 1, 1), (320, 64, 256, 1, 0), (512, 128, 256, 2, 1),
    (512, 0, 192, 2, 1), (640, 0, 64, 2, 1), (896, 448, 448, 2, 1)])
def test_both_block_forms_against_float64(pkg, torch_cuda, H, d_h, S, q_start, q_rows, split, causal):
    few = H * split * ((q_rows + 127) // 128) <= 148
    assert form(pkg, H, d_h, S, q_start, q_rows, split, causal) == ("128" if few else "tiles" if d_h < 64 else "256")
    check_against_float64(pkg, torch_cuda, H, d_h, S, q_start, q_rows, split, causal)


# Seven to 32 key stages, more than any ring of K/V slots holds: 256-row items whose two tiles have the same number of stages,
# one more in the second, or 64 rows in the second; 128-row items whose warpgroups get an odd and an even number.
@pytest.mark.parametrize("d_h", [16, 32, 64, 128])
@pytest.mark.parametrize("H,S,q_start,q_rows,split,causal,want", [
    (80, 1024, 768, 256, 1, 0, "256"), (90, 1600, 1344, 256, 1, 1, "256"), (76, 1024, 832, 192, 1, 0, "256"),
    (40, 3584, 3264, 256, 2, 1, "256"), (100, 1024, 960, 64, 1, 1, "128"), (5, 4096, 2880, 1216, 1, 1, "128"),
    (18, 2176, 64, 448, 2, 0, "128")])
def test_rings_that_wrap_against_float64(pkg, torch_cuda, d_h, H, S, q_start, q_rows, split, causal, want):
    assert form(pkg, H, d_h, S, q_start, q_rows, split, causal) == want
    check_against_float64(pkg, torch_cuda, H, d_h, S, q_start, q_rows, split, causal)


@pytest.mark.parametrize("d_h", [16, 32, 64, 128])
@pytest.mark.parametrize("tile_rows", [64, None])
@pytest.mark.parametrize("H,q_start,q_rows,split", [(50, 64, 704, 1), (50, 0, 576, 1), (19, 2048, 2048, 1), (38, 0, 1024, 2),
                                                    (100, 64, 704, 1), (120, 0, 576, 1), (60, 128, 448, 3)])
def test_a_short_last_wave(pkg, torch_cuda, d_h, H, q_start, q_rows, split, tile_rows):
    """Launches whose last wave is at most half full: from two full waves on (the last four shapes; at d_h 128 from one)
    its 256-row items go as 128-row ones, last blocks of 192 and 64 rows among them, of which the second half has 64 rows
    or none; below that the whole launch goes as 128-row items."""
    S = 4096 * split
    items = H * split * ((q_rows + 255) // 256)
    assert form(pkg, H, d_h, S, q_start, q_rows, split, 0) == ("256+128" if items > 296 or d_h == 128 else "128")
    check_against_float64(pkg, torch_cuda, H, d_h, S, q_start, q_rows, split, 0, growing=False, tile_rows=tile_rows)


@pytest.mark.parametrize("entry,d_h", [("forward", 16), ("forward", 32), ("noalloc", 16), ("noalloc", 64), ("noalloc", 128)])
@pytest.mark.parametrize("H,S", [(2, 512), (100, 512), (80, 1024), (160, 448)])
def test_the_largest_weight_of_a_row_is_not_rounded(pkg, torch_cuda, entry, d_h, H, S):
    """One key in the first stage and, by 2^3 to 2^8 larger in weight, one two stages later; V is 1 for the later one
    only, so that O is its softmax weight. With the row maximum as the exponent offset that weight enters P*V as exactly
    1 and O is right to fp32; under an offset that has not followed, it is off by its rounding to fp16 (up to 2.4e-4)."""
    torch = torch_cuda
    q_rows = 256
    if H == 160 and d_h < 64:
        assert form(pkg, H, d_h, S, S - q_rows, q_rows, 1, 0) == "tiles"
    p = pkg.make_params(S, H * d_h, H, 64)
    Q, K, V = (torch.zeros(H, S, d_h, dtype=torch.float16, device="cuda") for _ in range(3))
    per_log2 = 1.0 / (p.flash_tc.scale * 1.4426950408889634)              # score units that are one power of two
    Q[:, :, 0] = (3.0 + torch.arange(S, device="cuda") % 128 * (4.5 / 128)) * per_log2 / 8
    K[:, :, 0] = -64.0
    K[:, 0, 0], K[:, 300, 0] = 8.0, 16.0
    V[:, 300] = 1.0
    if entry == "forward":
        O, _ = run_attention(pkg, torch, p, [Q, K, V], S - q_rows, q_rows, pkg.F32)
    else:
        O = torch.zeros(q_rows, H * d_h, dtype=torch.float32, device="cuda")
        pkg.flash_attn_tc_forward_noalloc(Q, K, V, O, S - q_rows, q_rows, p.flash_tc, o_dtype=pkg.F32)
        torch.cuda.synchronize()
    s = Q[0, S - q_rows:, :1].double() * K[0, :, 0].double()[None, :] * p.flash_tc.scale
    ref = torch.softmax(s, dim=-1)[:, 300]
    assert 2 ** -8 < float((1 / ref - 1).min()) < float((1 / ref - 1).max()) < 2 ** -2.9
    assert float((O.double() / ref[:, None] - 1).abs().max()) < 5e-6


# One row to a block (few rows), several with a ragged last block (1024 rows: three), and the most (from 2368 rows on).
@pytest.mark.parametrize("rows", [64, 576, 640, 1024, 2368, 2432])
@pytest.mark.parametrize("split,H,d_h", [(2, 3, 16), (5, 2, 64)])
def test_merge_of_partials_by_number_of_rows(pkg, torch_cuda, rows, split, H, d_h):
    """flash_attn_tc_combine alone, from given partials, with rows before and behind those that are merged."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows)
    ws = rows + 128
    O = torch.randn(split, ws, H, d_h, generator=g, device="cuda")
    m = torch.randn(split, ws, H, generator=g, device="cuda") * 4
    l = torch.rand(split, ws, H, generator=g, device="cuda") + 1
    m[0, ::3] = float("-inf")                                  # a split without keys
    l[0, ::3] = 0
    O[0, ::3] = 0
    fp = pkg.FlashParams(64 * split * 64, d_h, H, split, 0, 1.0)
    out = torch.full((rows, H * d_h), float("nan"), device="cuda")
    pkg.flash_attn_tc_combine(pkg.FlashPartials(O.data_ptr(), m.data_ptr(), l.data_ptr(), ws), out, 64, rows, fp, None, pkg.F32)
    torch.cuda.synchronize()
    w = torch.exp2(m.double() - m.double().amax(0))
    want = ((w[..., None] * O.double()).sum(0) / (w * l.double()).sum(0)[..., None])[64:64 + rows].reshape(rows, -1)
    # sums of `split` fp32 terms and weights from exp2f: a few units in the last place of the largest term
    assert bool(((out.double() - want).abs() <= 16 * 2 ** -24 * (1 + want.abs().max())).all())


# A share of the exponentials is a polynomial: of the four chains (d_h 16 to 64, items of 128 and 256 rows) columns 14 and 15 of every 16, at d_h 128 (both
# kinds of items) 6 and 7 of every eight; none of the kernel of one tile (100 heads of 32, 256 keys).
@pytest.mark.parametrize("S,H,d_h,split", [(512, 2, 128, 1), (4096, 13, 128, 1), (256, 4, 64, 1), (512, 2, 16, 1), (256, 2, 32, 2), (4096, 12, 64, 1),
                                            (1536, 30, 32, 1), (256, 100, 32, 1)])
def test_weights_over_the_whole_exponent_range(pkg, torch_cuda, S, H, d_h, split):
    """Scores spread over several hundred powers of two, so that most weights vanish, some of them below the smallest number;
    and a NaN in the keys reaches every row, whichever way its exponential is computed."""
    torch = torch_cuda
    p = pkg.make_params(S, H * d_h, H, 64, 2, split, 0)
    g = torch.Generator(device="cuda").manual_seed(S + d_h)
    dev = [torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) * f for f in (8, 8, 1)]
    O, _ = run_attention(pkg, torch, p, dev, 0, S, pkg.F32)
    for h in range(H):
        q, k, v = (x[h].double() for x in dev)
        want = torch.softmax(q @ k.T * p.flash_tc.scale, 1) @ v
        got = O.view(S, H, d_h)[:, h].double()
        # fp16 weights (2^-11 each) of values up to max |V|, fp32 scores of up to 2^9: 2^-24 * 2^9 in the exponent
        assert bool(((got - want).abs() <= (2 ** -11 + 2 ** -13) * v.abs().max()).all())
    for key in (S - 128 + 78, S - 128 + 79, S - 128 + 70, 5):  # both columns of a pair that goes the one way, and two that go the other (70: at d_h up to 64)
        bad = [x.clone() for x in dev]
        bad[1][:, key, 3] = float("nan")
        O, _ = run_attention(pkg, torch, p, bad, 0, S, pkg.F32)
        assert torch.isnan(O).all()


# Of the columns of 16, 8 to 15, one to a head and split: those of the polynomial (14 and 15, at d_h 128 6 and 7 of every eight) and others.
@pytest.mark.parametrize("S,H,d_h,items128", [(4096, 8, 128, False), (1024, 4, 128, True), (1024, 4, 32, True), (1024, 4, 16, True), (4096, 8, 64, False),
                                              (4096, 8, 32, False), (4096, 8, 16, False), (1024, 4, 64, True)])
def test_each_weight_is_as_exact_as_its_exponential(pkg, torch_cuda, S, H, d_h, items128):
    """Two keys per row and split carry weight, the maximum (weight 1) and one of 2^x, x from -1 to 0 over the rows: the fp32
    denominator shows the exponential itself, with one rounding."""
    torch = torch_cuda
    split = 2
    fp = pkg.FlashParams(S, d_h, H, split, 0, 1.0)
    plan = pkg.flash_attn_tc_plan(fp, 0, S)
    assert (plan.items_128 > 0) == items128 and (plan.items_256 > 0) != items128 and plan.tiles == 0
    g = torch.Generator(device="cuda").manual_seed(d_h)
    Q = torch.zeros(H, S, d_h, device="cuda", dtype=torch.float16)
    Q[..., 0] = (torch.rand(H, S, generator=g, device="cuda") * 0.69).half()
    Q[..., 1] = torch.randint(0, 1024, (H, S), generator=g, device="cuda").half() / 1024
    Q[..., 2] = 1
    K = torch.zeros(H, S, d_h, device="cuda", dtype=torch.float16)
    K[..., 2] = -1000                                           # no weight
    V = torch.zeros(H, S, d_h, device="cuda", dtype=torch.float16)
    column = torch.empty(split, H, dtype=torch.int64)
    for i in range(split):
        for h in range(H):
            # behind the maximum in the same chain: 64 keys further chains of 64 keys change, and the weight is one of their merge
            column[i, h] = (2 * h + i) % 8 + 8 + 16 * ((5 * h + 3 * i) % (8 if d_h == 128 else 4))
            K[h, i * (S // split) + 9, 2] = 0                   # score 0, in the first stage of 128 keys
            K[h, i * (S // split) + 256 + column[i, h], :3] = torch.tensor([-1, -2.0 ** -12, 0])
    ws = [torch.full((n,), float("nan"), device="cuda") for n in (split * S * H * d_h, split * S * H, split * S * H)]
    part = pkg.FlashPartials(*(w.data_ptr() for w in ws), S)
    pkg.flash_attn_tc_forward(Q, K, V, None, part, 0, S, fp, o_dtype=pkg.F32)
    torch.cuda.synchronize()
    m, l = ws[1].view(split, S, H), ws[2].view(split, S, H)
    assert bool((m == 0).all())
    score = -(Q[..., 0].float() + Q[..., 1].float() * 2.0 ** -12).T          # exact in fp32
    w = torch.exp2((score * 1.4426950408889634).double())                     # the argument rounded to fp32, as the kernel has it
    err = (l.double() - (1 + w)).abs()
    by_poly = (column % 16 >= 14 if d_h <= 64 else column % 8 >= 6).to(err.device)[:, None, :]
    assert {14, 15} <= {int(c) % 16 for c in column.flatten()}
    # the error stated for either way, and the rounding of a sum between 1 and 2
    bound = torch.where(by_poly, 1.8e-7, 2.0 ** -22) * w + 2.0 ** -24
    assert bool((err <= bound).all()), float((err - bound).max())
