"""The order in which causal attention launches without counters take their work items: every item once, longest first, whatever the
numbers (the function itself, compiled for the CPU); and the same bits as a launch that takes its rows in plain order."""
import ctypes
import os
import random
import subprocess

import pytest

from conftest import ROOT

SOURCE = """
#include "work_order.h"
extern "C" void items(int n, int heads, int splits, int blocks, int group, int split_blocks, int* out)
{
    for (int u = 0; u < n; u++) efa::grouped_item(u, heads, splits, blocks, group, split_blocks, out[3 * u], out[3 * u + 1], out[3 * u + 2]);
}
"""


@pytest.fixture(scope="module")
def items(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "order.cpp").write_text(SOURCE)
    so = d / "order.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "eager-flash-attention_b200", "csrc"),
                    str(d / "order.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def run(heads, splits, blocks, group, split_blocks):
        n = heads * splits * blocks
        out = (ctypes.c_int * (3 * n))()
        lib.items(n, heads, splits, blocks, group, split_blocks, out)
        return [tuple(out[3 * i:3 * i + 3]) for i in range(n)]
    return run


def _shapes():
    rng = random.Random(5)
    yield from [(1, 1, 1, 1, 1), (16, 1, 64, 16, 64), (4, 4, 64, 4, 16), (3, 16, 1, 2, 1), (5, 2, 1, 5, 64), (7, 3, 4, 3, 9), (2, 8, 9, 2, 1)]
    for _ in range(200):
        heads = rng.randint(1, 9)
        yield heads, rng.randint(1, 16), rng.randint(1, 20), rng.randint(1, heads), rng.randint(1, 24)


def test_every_item_comes_once_and_groups_follow_one_another(items):
    for heads, splits, blocks, group, split_blocks in _shapes():
        got = items(heads, splits, blocks, group, split_blocks)
        assert sorted(got) == [(h, s, b) for h in range(heads) for s in range(splits) for b in range(blocks)]
        of_group = [h // group for h, _, _ in got]
        assert of_group == sorted(of_group)


def test_longest_items_first(items):
    """Keys of an item of one row block: those of its split up to the last row of the block."""
    for heads, splits, blocks, group, split_blocks in _shapes():
        got = items(heads, splits, blocks, group, split_blocks)
        for g in range(0, heads, group):
            keys = [min(split_blocks, max(0, b + 1 - s * split_blocks)) for h, s, b in got if h // group == g // group]
            assert keys == sorted(keys, reverse=True)


@pytest.mark.gpu
# heads that fill no whole group (64 MB of K and V), one head to a group, 256- and 128-row items, splits with empty items, rows that start
# inside the sequence, a split that is no multiple of an item's rows, all head sizes
@pytest.mark.parametrize("S,H,d_h,split,q_start,q_rows", [(16384, 9, 128, 1, 8192, 8192), (65536, 3, 128, 1, 65536 - 4096, 4096), (4096, 3, 64, 1, 0, 4096),
                                                          (4096, 5, 64, 4, 0, 4096), (4032, 7, 64, 3, 64, 2624), (960, 2, 64, 5, 0, 960),
                                                          (2048, 16, 32, 2, 0, 2048), (4096, 24, 16, 1, 0, 4096), (8192, 6, 32, 1, 0, 8192),
                                                          (4096, 4, 128, 8, 2048, 2048)])
def test_same_bits_as_in_row_order(pkg, torch_cuda, S, H, d_h, split, q_start, q_rows):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + H)
    q, k, v = (torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))
    p = pkg.FlashParams(S, d_h, H, split, 1, d_h ** -0.5)
    ws = [torch.full((n,), float("nan"), device="cuda") for n in (split * q_rows * H * d_h, split * q_rows * H, split * q_rows * H)]
    part = pkg.FlashPartials(*(w.data_ptr() for w in ws), q_rows) if split > 1 else None
    got = []
    for counters in (None, torch.zeros((q_rows + 63) // 64, dtype=torch.int32, device="cuda")):
        out = torch.full((q_rows, H * d_h), float("nan"), dtype=torch.float16, device="cuda")
        for w in ws:
            w.fill_(float("nan"))
        pkg.kernel_status_reset()
        pkg.flash_attn_tc_forward(q, k, v, out, part, q_start, q_rows, p, tile_counters=counters, tile_rows=64 if counters is not None else 0, o_dtype=pkg.F16)
        if part is not None:
            pkg.flash_attn_tc_combine(part, out, 0, q_rows, p, o_dtype=pkg.F16)
        torch.cuda.synchronize()
        assert pkg.kernel_status()[0] == 0
        got.append([out] + ([w.clone() for w in ws] if split > 1 else []))
    for a, b in zip(*got):
        assert torch.isfinite(a).all() or split > 1
        assert torch.equal(torch.nan_to_num(a, 7.0), torch.nan_to_num(b, 7.0))
