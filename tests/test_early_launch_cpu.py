"""Kernels that may be on the GPU before the kernel ahead of them has ended (launch_early) read memory that is still being
written when they start. Loads that presume read-only memory are no option for them: the sources are looked through."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "eager-flash-attention_b200", "csrc")


def _sources():
    text = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        with open(path) as f:
            text[path] = re.sub(r"//[^\n]*", "", f.read())
    return text


def _definition(text, name):
    """Parameters and body of the kernel `name`, or None."""
    at = re.search(r"__global__[^;{]*?\b" + name + r"\(", text)
    if not at:
        return None
    depth, i = 0, text.index("{", at.end())
    for k in range(i, len(text)):
        depth += (text[k] == "{") - (text[k] == "}")
        if depth == 0:
            return text[at.start():k + 1]
    raise AssertionError(f"{name}: no end")


def _early_kernels():
    sources = _sources()
    names = {n for text in sources.values() for n in re.findall(r"launch_(?:early|early_cluster|kernel)\((?:\w+,\s*)*(\w+_kernel)\b", text)}
    found = {}
    for name in names:
        bodies = [b for b in (_definition(text, name) for text in sources.values()) if b]
        assert len(bodies) == 1, name                       # two kernels of one name could not be told apart
        found[name] = bodies[0]
    return found


def test_kernels_that_start_early_are_found():
    assert set(_early_kernels()) == {"combine_splits_kernel", "fa_fwd_ws_kernel", "fa_fwd_chains_kernel", "fa_fwd_tile_kernel", "proj_gemm_kernel",
                                     "proj_pair_kernel", "proj_tile_kernel", "proj_split_kernel"}


def test_kernels_have_names_of_their_own():
    """Profiles and launch lists tell kernels apart by name."""
    names = [n for text in _sources().values() for n in re.findall(r"__global__\s+void\s+(?:__\w+__\s*\([^)]*\)\s*)*(\w+)\s*\(", text)]
    assert {"fa_fwd_ws_kernel", "combine_splits_kernel"} < set(names) and len(names) == len(set(names)), sorted(names)


def test_kernels_that_start_early_presume_no_read_only_memory():
    for name, body in _early_kernels().items():
        assert body, name
        assert not re.search(r"__restrict__|__ldg\b|\.nc\b|__constant__", body), name
        assert "pdl_wait()" in body and "pdl_trigger()" in body, name


def test_helpers_that_kernels_share_presume_no_read_only_memory():
    for name in ("sm100_ptx.cuh", "fa_args.cuh", "work_order.h"):
        with open(os.path.join(CSRC, name)) as f:
            assert not re.search(r"__restrict__|__ldg\b|global\.nc\b", f.read())


def test_an_order_table_is_not_read_while_it_may_be_written():
    """order_tab, which pick_item reads, is device memory. A kernel that picks its item ahead of pdl_wait() is not launched early with a table."""
    kernels = {name: body for name, body in _early_kernels().items() if re.search(r"\bpick_item\(|order_tab", body)}
    assert set(kernels) == {"fa_fwd_ws_kernel", "fa_fwd_chains_kernel"}
    text = "".join(_sources().values())
    for name, body in kernels.items():
        body = re.sub(r"auto (\w+) = \[&\]\([^)]*\)(?: -> \w+)? \{.*?\n    \};", "", body, flags=re.S)     # what they define is judged where it is called
        ahead = re.search(r"\b(?:fetch_item|pick_item)\(", body.split("pdl_wait()", 1)[0])
        launches = re.findall(r"launch_(early|kernel)\((?:(\w+), \d, )?" + name + "<", text)
        assert launches
        if ahead:
            assert set(launches) == {("kernel", "early")}, name
            assert text.count("const bool early = args.order_tab == nullptr;") == len(launches), name
