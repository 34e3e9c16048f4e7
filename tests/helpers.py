"""Shared test helpers: golden-fixture loading and conversions between stored 16-bit patterns, numpy and torch."""
from pathlib import Path

import numpy as np

GOLDEN = Path(__file__).resolve().parent / "golden"

PREFILL_GOLDENS = ["p_gqa_small", "p_mha_tail", "p_mqa_multi", "p_k9", "p_one_chunk", "p_gqa_256", "p_fp16_gqa", "p_fp16_d128"]
DECODE_GOLDENS = ["d_small", "d_d128", "d_mha", "d_fp16"]
ROUTE_GOLDENS = ["r_upstream_gqa", "r_upstream_mqa"]


class HalfBits(np.ndarray):
    """uint16 bit patterns of IEEE half values (plain uint16 arrays in a fixture are bf16 patterns)."""


def load(name):
    """The fixture as a dict; the 16-bit inputs of a fixture whose `dtype` entry says float16 come back as HalfBits,
    so that bits_to_f64 / bits_to_torch decode them in the right format."""
    g = dict(np.load(GOLDEN / f"{name}.npz"))
    if str(g.get("dtype", "bfloat16")) == "float16":
        for key, value in g.items():
            if value.dtype == np.uint16:
                g[key] = value.view(HalfBits)
    return g


def unpack_selected(g, tag):
    """[F,Hq,T] bool selection stored bit-packed as selected_<tag>_packed + selected_shape."""
    shape = g["selected_shape"]
    return np.unpackbits(g[f"selected_{tag}_packed"])[:int(np.prod(shape))].reshape(shape).astype(bool)


def bits_to_f64(bits):
    """uint16 bit patterns (bf16, or half when tagged HalfBits) -> float64 values."""
    if isinstance(bits, HalfBits):
        return np.asarray(bits).view(np.float16).astype(np.float64)
    return (np.asarray(bits, dtype=np.uint16).astype(np.uint32) << 16).view(np.float32).astype(np.float64)


def bits_to_torch(bits, device="cpu"):
    import torch
    dtype = torch.float16 if isinstance(bits, HalfBits) else torch.bfloat16
    t = torch.from_numpy(np.asarray(bits, dtype=np.uint16).view(np.int16).copy()).view(dtype)
    return t.to(device)


def torch_to_f64(t):
    return t.detach().float().cpu().numpy().astype(np.float64)


def cu_from_lens(lens):
    return np.concatenate(([0], np.cumsum(np.asarray(lens, dtype=np.int64))))


def rel_rms(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return float(np.sqrt(((a - b) ** 2).mean()) / max(np.sqrt((b ** 2).mean()), 1e-30))


def config1_inputs():
    """BASELINE config 1 inputs: seed 0, q, k, v then dO ~ N(0,1), [2048, 8, 64], rounded to bf16."""
    import torch
    rng = torch.Generator().manual_seed(0)
    q, k, v = [torch.randn(2048, 8, 64, generator=rng).bfloat16() for _ in range(3)]
    g = torch.randn(2048, 8, 64, generator=rng).bfloat16()
    return q, k, v, g


def two_threads(calls, times=20000):
    """Runs each (entry point, arguments) `times` times in a thread of its own, both at once: how many of each failed."""
    import threading

    import torch
    failed, start = [0] * len(calls), threading.Barrier(len(calls))

    def loop(i):
        entry, args = calls[i]
        start.wait()
        for _ in range(times):
            failed[i] += entry(*args) != 0
    threads = [threading.Thread(target=loop, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return failed


# MOBA_ATTEND_* of the library's header: the decode attention kernels
FIXED_DEEP, FIXED, STREAMED, CLUSTER_8, CLUSTER_16 = 1, 2, 3, 8, 16


def attend_kernels(cache):
    """A list that grows by the kernel of every attention that `cache` launches from now on, as the library answers for the
    arguments of that launch."""
    taken, launch = [], cache._launch

    def recorded(name, *args):
        if name == "moba_decode_attend":
            desc, rows, hq, selected, slots, umax = args[0], args[4], args[5], args[6], args[7], args[11]
            taken.append(cache._lib.moba_decode_attend_variant(desc, rows, hq, int(selected is not None), slots, umax, 0, -1))
        return launch(name, *args)
    cache._launch = recorded
    return taken
