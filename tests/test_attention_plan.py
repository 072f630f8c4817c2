"""Which items a causal attention launch goes as: 128-row items where its longest 256-row item is what it takes, on the CPU; and the results of
launches on both sides of that line, on the GPU."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

SOURCE = """
#include "attention_plan.h"
extern "C" void plan(int q_start, int q_rows, int S, int H, int split, int causal, int d_h, int longest_first, int* out)
{
    const efa::FaPlan p = efa::plan_items(efa::PlanShape{q_start, q_rows, S, H, split, S / split, causal, d_h, true, longest_first != 0, 148});
    out[0] = p.items256; out[1] = p.items128; out[2] = p.tiles;
}
"""


@pytest.fixture(scope="module")
def plan_items(tmp_path_factory):
    """The arithmetic of the plan, compiled for the CPU: (items of 256 rows, of 128 rows, tiles)."""
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "eager-flash-attention_b200", "csrc"),
                    str(d / "plan.cpp"), "-o", str(d / "plan.so")], check=True)
    lib = ctypes.CDLL(str(d / "plan.so"))

    def run(*args):
        out = (ctypes.c_int * 3)()
        lib.plan(*args, out)
        return tuple(out)
    return run


@pytest.mark.parametrize("d_h,S,H,q_start,split,halves", [
    (64, 4096, 8, 0, 1, True), (128, 8192, 4, 0, 1, True), (64, 1024, 32, 0, 1, True), (128, 1024, 32, 0, 1, False), (64, 2048, 20, 0, 1, True),
    (64, 2048, 24, 0, 1, False), (128, 2048, 20, 0, 1, False), (64, 512, 64, 0, 1, False), (64, 4096, 8, 0, 2, False), (64, 16384, 16, 0, 1, False),
    (64, 8192, 37, 7168, 1, False), (32, 4096, 8, 0, 1, True)])
def test_items_under_a_mask(pkg, d_h, S, H, q_start, split, halves):
    plan = pkg.flash_attn_tc_plan(pkg.FlashParams(S, d_h, H, split, 1, 1.0), q_start, S - q_start)
    assert plan.tiles == 0 and (plan.items_128 > 0) == halves and (plan.items_256 > 0) != halves
    assert plan.stage_step == (2 if halves else 1)


# With completion counters the rows go in order, and the longest item is the last to start.
@pytest.mark.parametrize("d_h,S,H,q_start,longest_first,in_order", [
    (128, 4096, 8, 0, True, False), (128, 8192, 4, 2048, True, False), (128, 2048, 12, 0, True, False), (128, 1024, 24, 0, True, False), (128, 4096, 5, 0, True, True),
    (128, 8192, 3, 0, True, True), (128, 3072, 20, 1536, False, False), (64, 768, 32, 0, True, False), (64, 4096, 8, 0, True, True), (32, 4096, 20, 2048, False, True),
    (64, 65536, 1, 0, False, True), (64, 41216, 3, 0, False, False), (16, 1536, 48, 384, False, False),
    (64, 640, 40, 128, True, False)])
def test_items_under_a_mask_by_the_order_of_the_launch(plan_items, d_h, S, H, q_start, longest_first, in_order):
    for first, halves in ((1, longest_first), (0, in_order)):
        items256, items128, tiles = plan_items(q_start, S - q_start, S, H, 1, 1, d_h, first)
        assert ((items256 > 0), (items128 > 0), tiles) == (not halves, halves, 0), first


# By waves: of 256-row items against those of tiles, two to an SM; under a mask where items are of about one length or tiles more than a wave.
@pytest.mark.parametrize("S,H,causal,item_rows", [(640, 50, 0, 0), (640, 110, 0, 0), (640, 60, 0, 256), (640, 160, 0, 256), (384, 160, 0, 0), (384, 250, 0, 0), (384, 200, 0, 256),
                                             (576, 160, 0, 256), (512, 148, 0, 256), (896, 60, 1, 256), (896, 75, 1, 0), (768, 75, 1, 256), (640, 75, 1, 0)])
def test_few_keys_by_waves(plan_items, S, H, causal, item_rows):
    if causal:          # a window of the last rows: items of 4.25 to 6 stages
        assert plan_items(320, 320, 640, 90, 1, 1, 32, 1) == plan_items(320, 320, 640, 90, 1, 1, 32, 0) == (0, 0, 270)
        assert plan_items(512, 128, 640, 190, 1, 1, 16, 0) == (0, 0, 190) and plan_items(128, 640, 768, 50, 1, 1, 16, 1) == (150, 0, 0)
    want = (0, 0, H * ((S + 127) // 128)) if item_rows == 0 else (H * ((S + 255) // 256), 0, 0)
    assert plan_items(0, S, S, H, 1, causal, 32, 1) == want


@pytest.mark.parametrize("d_h,S,H,causal,slots,step", [(16, 128, 592, 0, 2, 1), (16, 256, 200, 1, 2, 1), (32, 384, 200, 0, 4, 1), (32, 512, 128, 1, 2, 1), (32, 512, 64, 1, 4, 1), (16, 640, 75, 1, 2, 1), (16, 768, 100, 1, 4, 1),
                                                       (32, 384, 148, 0, 4, 1), (32, 384, 222, 0, 4, 1),
                                                       (16, 2048, 16, 1, 4, 2), (32, 1024, 32, 1, 4, 2), (32, 640, 160, 0, 4, 1)])
def test_tiles_of_few_keys(pkg, d_h, S, H, causal, slots, step):
    """Blocks of their own (two slots) up to two stages of keys, or five in uneven waves; items of 256 or 128 rows (four slots) above that. The plan
    names what is launched."""
    plan = pkg.flash_attn_tc_plan(pkg.FlashParams(S, d_h, H, 1, causal, 1.0), 0, S)
    tiles, items256 = H * S // 128, H * ((S + 255) // 256)
    assert (plan.items_256, plan.items_128, plan.tiles) == ((0, 0, tiles) if slots == 2 else (items256, 0, 0) if step == 1 else (0, tiles, 0))
    assert (plan.k_slots, plan.v_slots, plan.stage_step) == (slots, slots, step)


@pytest.mark.gpu
@pytest.mark.parametrize("d_h,S,H,causal", [(64, 2048, 20, 1), (128, 4096, 8, 1), (32, 1024, 32, 1), (16, 384, 200, 0), (32, 640, 160, 1), (16, 256, 200, 1)])
def test_results(pkg, torch_cuda, d_h, S, H, causal):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + H)
    q, k, v = (torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))
    fp = pkg.FlashParams(S, d_h, H, 1, causal, d_h ** -0.5)
    out = torch.full((S, H * d_h), float("nan"), device="cuda")
    pkg.kernel_status_reset()
    pkg.flash_attn_tc_forward(q, k, v, out, None, 0, S, fp, o_dtype=pkg.F32)
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0
    for h in range(0, H, 7):
        s = q[h].double() @ k[h].double().T * d_h ** -0.5
        if causal:
            s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
        w = torch.softmax(s, dim=-1)
        ref = w @ v[h].double()
        # every weight is rounded to fp16 (2^-11 of it) or, below 2^-14 of the largest, to a multiple of 2^-25 (the offset may lag the
        # maximum by 2^8); fp32 scores of up to about 100 carry 1e-5 of relative error into the weights
        bound = (w * 2 ** -11 + 2.0 ** -24) @ v[h].double().abs() + 1e-4 * ref.abs().max()
        assert bool(((out[:, h * d_h:(h + 1) * d_h].double() - ref).abs() <= bound).all()), h
