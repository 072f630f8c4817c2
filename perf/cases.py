"""What a user of this library has it do, as cases that can be timed and compared.

A case is one call (or the pair of calls that belong together) through the public interface of the package: the
attention launch interface, the projection, the Q/K/V projections before the block, and whole blocks through the run
modes, on device and on host buffers. Sizes are those of the library's own benchmark, its configurations and tests.
"""
import importlib
import math

import torch

efa = importlib.import_module("eager-flash-attention_b200")

_MODES = {"stream": efa.MODE_STREAM, "megatron": efa.MODE_MEGATRON, "overlap": efa.MODE_OVERLAP}
_ctx = None


def _context():
    """Streams and communicators: one per process, as every program of this library keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = efa.make_ctx(efa.World(), ncomm=4)
    return _ctx


def _block(name, mode, S, H, d_h, tile, causal, split=1, host=False, f32=False):
    return dict(name=name, kind="block", mode=mode, S=S, H=H, d_h=d_h, tile=tile, causal=causal, split=split, host=host, f32=f32)


def _attn(name, S, H, d_h, causal, split=1, q_start=0, q_rows=0, o32=False, tile=0, noalloc=False):
    """q_rows = 0: all rows. tile > 0: with completion counters of that many rows. noalloc: the entry without a workspace."""
    return dict(name=name, kind="attention", S=S, H=H, d_h=d_h, causal=causal, split=split, q_start=q_start,
                q_rows=q_rows or S - q_start, o32=o32, tile=tile, noalloc=noalloc)


def listed():
    return [
        # Whole blocks on one GPU (attention, output projection, reduction), the interface that programs call.
        # The smallest: a shape of the correctness matrix, where launches and host work are the time.
        _block("block_small", "stream", 1024, 8, 64, 256, True),
        # The single-GPU configuration of the benchmark plan, tile by tile behind one attention launch.
        _block("block_4k", "stream", 4096, 16, 64, 128, False),
        # The one-shot mode at the sequence length of the sweep suites.
        _block("block_16k_megatron", "megatron", 16384, 16, 64, 2048, True),
        # The benchmark itself, and the largest.
        _block("block_32k", "stream", 32768, 32, 128, 128, True),
        # A block on pinned host buffers: copy-in, compute and copy-out of one call.
        _block("block_host_8k", "stream", 8192, 32, 128, 128, True, host=True),
        # The attention launch of one of eight ranks, long sequence, with the completion counters a consumer waits on.
        _attn("attn_64k_2heads", 65536, 2, 64, False, tile=128),
        # One of eight ranks of the benchmark: four heads of 128.
        _attn("attn_32k_4heads", 32768, 4, 128, True),
        # One of four ranks of the sweep suites: split-KV and the merge after it.
        _attn("attn_16k_split4", 16384, 4, 64, True, split=4),
        # Small heads and the fp32 output of the original launch interface; an odd multiple of 64 rows.
        _attn("attn_d32_f32", 4032, 8, 32, False, o32=True),
        # One 128-row tile against a long context without a workspace: the latency-critical call.
        _attn("attn_tile_noalloc", 16384, 16, 64, False, split=8, q_start=8192, q_rows=128, noalloc=True),
        # The projection of a group of rows of one of eight ranks, with a ragged last tile.
        dict(name="project_ragged", kind="project", rows=4160, d_local=512, d=4096),
        # The Q/K/V projections before the block, one of eight ranks of the benchmark.
        dict(name="qkv_8k_4heads", kind="qkv", S=8192, d=4096, H=4, d_h=128),
    ]


def _log(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], spread over its logarithm."""
    lo, hi = -(-lo // step) * step, hi // step * step
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def _draw_once(rng):
    kind = rng.choice(["block", "block", "attention", "attention", "attention", "noalloc", "project", "qkv"])
    if kind == "block":
        d_h = rng.choice([64, 64, 128, 32])
        H = rng.choice([4, 8, 16, 32])
        tile = rng.choice([64, 128, 256, 512])
        split = rng.choice([1, 1, 1, 2, 4])
        S = _log(rng, 512, 32768, math.lcm(tile, 64 * split))
        mode = rng.choice(["stream", "stream", "megatron", "overlap"])
        host = mode == "stream" and S * H * d_h <= 8192 * 4096 and rng.random() < 0.25
        f32 = not host and rng.random() < 0.2
        c = _block(None, mode, S, H, d_h, tile, True if host else rng.random() < 0.5, split, host, f32)
    elif kind == "project":
        c = dict(kind="project", rows=_log(rng, 64, 32768, 64), d_local=_log(rng, 64, 4096, 16), d=_log(rng, 256, 4096, 64))
    elif kind == "qkv":
        d_h = rng.choice([64, 128])
        c = dict(kind="qkv", S=_log(rng, 512, 32768, 64), d=_log(rng, 256, 4096, 64), H=rng.choice([1, 2, 4, 8, 16]), d_h=d_h)
    else:
        d_h = rng.choice([16, 32, 64, 64, 128, 128])
        H = rng.choice([1, 2, 3, 4, 8, 16, 32])
        split = rng.choice([1, 1, 2, 4, 8]) if kind == "attention" else rng.choice([1, 2, 4, 8])
        S = _log(rng, 256, 65536, 64 * split)
        q_start, q_rows = 0, S
        if kind == "noalloc":
            q_rows = min(S, rng.choice([64, 128, 192, 512]))
        elif rng.random() < 0.25:
            q_rows = _log(rng, 64, S, 64)
        if q_rows < S:
            q_start = 64 * rng.randint(0, (S - q_rows) // 64)
        tile = rng.choice([64, 128, 256]) if kind == "attention" and rng.random() < 0.5 else 0
        c = _attn(None, S, H, d_h, rng.random() < 0.5, split, q_start, q_rows, rng.random() < 0.3, tile, kind == "noalloc")
        if c["noalloc"] and split > 1 and split * q_rows * (H * d_h + 2 * H) * 4 > efa.STATIC_SCRATCH_BYTES:
            return None
    c.pop("name", None)
    return c


def draw(rng):
    most = work(_block(None, "stream", 32768, 32, 128, 128, True))
    while True:
        c = _draw_once(rng)
        # small heads take longer per operation than large ones: at most a sixteenth of the largest case's operations
        if c and work(c)["flops"] * (16 if c.get("d_h", 128) < 64 else 2 if c.get("d_h", 128) < 128 else 1) <= most["flops"]:
            return c


def _flash_params(S, H, d_h, split, causal):
    return efa.FlashParams(S, d_h, H, split, int(causal), 1.0 / math.sqrt(d_h))


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, sigma=1.0):
        x = torch.randn(*shape, generator=g, device="cuda", dtype=torch.float16)
        return x if sigma == 1.0 else x.mul_(sigma)

    k = case["kind"]
    s = dict(case=case)
    if k == "project":
        s.update(A=normal(case["rows"], case["d_local"]), W=normal(case["d_local"], case["d"], sigma=case["d"] ** -0.5),
                 out=torch.empty(case["rows"], case["d"], dtype=torch.float16, device="cuda"))
    elif k == "qkv":
        S, d, H, d_h = (case[n] for n in ("S", "d", "H", "d_h"))
        s.update(X=normal(S, d), W=[normal(H, d, d_h, sigma=d ** -0.5) for _ in range(3)],
                 out=[torch.empty(H, S, d_h, dtype=torch.float16, device="cuda") for _ in range(3)])
    elif k == "attention":
        S, H, d_h, split, rows = (case[n] for n in ("S", "H", "d_h", "split", "q_rows"))
        s.update(qkv=[normal(H, S, d_h) for _ in range(3)], fp=_flash_params(S, H, d_h, split, case["causal"]),
                 dtype=efa.F32 if case["o32"] else efa.F16, part=None, counters=None,
                 O=torch.empty(rows, H * d_h, dtype=torch.float32 if case["o32"] else torch.float16, device="cuda"))
        if split > 1 and not case["noalloc"]:
            ws = [torch.empty(n, dtype=torch.float32, device="cuda") for n in (split * rows * H * d_h, split * rows * H, split * rows * H)]
            s.update(ws=ws, part=efa.FlashPartials(*(w.data_ptr() for w in ws), rows))
        if case["tile"]:
            s["counters"] = torch.zeros((rows + case["tile"] - 1) // case["tile"], dtype=torch.int32, device="cuda")
    else:
        S, H, d_h = (case[n] for n in ("S", "H", "d_h"))
        d = H * d_h
        p = efa.make_params(S, d, H, case["tile"], split=case["split"], causal=case["causal"])
        p.proj_f32 = int(case["f32"])
        t = [normal(H, S, d_h) for _ in range(3)] + [normal(d, d, sigma=d ** -0.5)]
        odt = torch.float32 if case["f32"] else torch.float16
        if case["host"]:
            t = [x.cpu().pin_memory() for x in t]
            s["out"] = torch.empty(S, d, dtype=odt, pin_memory=True)
        else:
            s["out"] = torch.empty(S, d, dtype=odt, device="cuda")
            s["weights"] = efa.Weights(*(x.data_ptr() for x in t))
        s.update(tensors=t, p=p, ctx=_context(), mode=_MODES[case["mode"]])
        torch.cuda.synchronize()        # the run modes work on streams of their own
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "project":
        efa.project(s["A"], s["W"], s["out"], case["rows"], case["d_local"], case["d"])
        return s["out"]
    if k == "qkv":
        efa.compute_qkv(s["X"], *s["W"], *s["out"], case["S"], case["d"], case["H"], case["d_h"])
        return s["out"]
    if k == "attention":
        Q, K, V = s["qkv"]
        if case["noalloc"]:
            efa.flash_attn_tc_forward_noalloc(Q, K, V, s["O"], case["q_start"], case["q_rows"], s["fp"], o_dtype=s["dtype"])
            return s["O"]
        if s["counters"] is not None:
            s["counters"].zero_()
        efa.flash_attn_tc_forward(Q, K, V, s["O"], s["part"], case["q_start"], case["q_rows"], s["fp"],
                                  tile_counters=s["counters"], tile_rows=case["tile"], o_dtype=s["dtype"])
        if s["part"] is not None:
            efa.flash_attn_tc_combine(s["part"], s["O"], 0, case["q_rows"], s["fp"], o_dtype=s["dtype"])
        return s["O"] if s["counters"] is None else (s["O"], s["counters"])
    if case["host"]:
        efa.run_mode_host(s["ctx"], s["mode"], *s["tensors"], s["out"], s["p"])
    else:
        efa.run_mode(s["ctx"], s["mode"], s["weights"], s["out"], s["p"])
    return s["out"]


def _attention_flops(S, H, d_h, causal, q_start, q_rows):
    """Q K^T and P V over the keys that the rows may see."""
    pairs = q_rows * (2 * q_start + q_rows + 1) / 2 if causal else q_rows * S
    return 4.0 * pairs * d_h * H


def work(case):
    k = case["kind"]
    if k == "project":
        m, n, kk = case["rows"], case["d"], case["d_local"]
        return {"bytes": 2.0 * (m * kk + kk * n + m * n), "flops": 2.0 * m * n * kk}
    S, H, d_h = (case[n] for n in ("S", "H", "d_h"))
    d = H * d_h
    if k == "qkv":
        kk = case["d"]
        return {"bytes": 2.0 * (S * kk + 3 * kk * d + 3 * S * d), "flops": 2.0 * S * kk * 3 * d}
    if k == "attention":
        rows, keys = case["q_rows"], case["q_start"] + case["q_rows"] if case["causal"] else S
        return {"bytes": 2.0 * d * (rows + 2 * keys) + (4.0 if case["o32"] else 2.0) * rows * d,
                "flops": _attention_flops(S, H, d_h, case["causal"], case["q_start"], rows)}
    return {"bytes": 2.0 * (3 * S * d + d * d) + (4.0 if case["f32"] else 2.0) * S * d,
            "flops": _attention_flops(S, H, d_h, case["causal"], 0, S) + 2.0 * S * d * d}


def tolerance(case):
    """fp16 operands (the softmax weights among them) and fp16 results, fp32 sums. Against the same path in 64 bits the
    cases and two dozen drawn ones are off by up to 3.6e-4 (2-norm) and 3.7e-3 (largest difference): four times that."""
    return {"rel": 1.4e-3, "max": 1.5e-2}
