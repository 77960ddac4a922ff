"""Calls of C entry points without ctypes (csrc/hostcall.cc): what arrives is what was handed over, whatever the mix of
integers, addresses and floats."""

import ctypes
import random

import pytest
import torch

from enginekernel_b200.ops import lib
from enginekernel_b200.parts.base import Workspace

TYPES = {"p": ctypes.c_void_p, "i": ctypes.c_int, "q": ctypes.c_longlong, "f": ctypes.c_float}


@pytest.mark.parametrize("seed", range(12))
def test_arguments_arrive(seed):
    host = lib._host_module()
    if not host:
        pytest.skip("no C++ compiler or no headers of this interpreter")
    rng = random.Random(seed)
    floats = rng.randint(0, 8)
    kinds = ["f"] * floats + [rng.choice("piq") for _ in range(rng.choice([0, 1, 5, 6, 7, 20, 48]))]
    rng.shuffle(kinds)
    seen = []

    def record(*args):
        seen.append(args)
        return seed - 5
    proto = ctypes.CFUNCTYPE(ctypes.c_int, *[TYPES[k] for k in kinds])
    target = proto(record)
    call = host.bind(ctypes.cast(target, ctypes.c_void_p).value, "".join("i" if k == "q" else k for k in kinds))
    t = torch.zeros(3)
    args, want = [], []
    for k in kinds:
        if k == "f":
            v = rng.choice([0.0, -1.5, 3, 1e-30])
            args.append(v), want.append(ctypes.c_float(v).value)
        elif k == "p":
            v = rng.choice([None, t, rng.randrange(1, 1 << 62)])
            args.append(v), want.append(t.data_ptr() if v is t else v)
        else:
            v = rng.choice([0, -1, True, rng.randrange(-(1 << 31), 1 << 31) if k == "i" else rng.randrange(-(1 << 63), 1 << 63)])
            args.append(v), want.append(int(v))
    assert call(*args) == seed - 5 and list(seen[0]) == want
    with pytest.raises(TypeError):
        call(*args, 1)
    for at, k in enumerate(kinds):
        with pytest.raises((TypeError, AttributeError)):
            call(*args[:at], "text", *args[at + 1:])
    assert len(seen) == 1


def test_other_signatures_stay_with_ctypes():
    host = lib._host_module()
    if not host:
        pytest.skip("no C++ compiler or no headers of this interpreter")
    assert host.bind(1, "f" * 9) is None and host.bind(1, "i" * 49) is None and host.bind(1, "d") is None
    assert host.bind(1, "f" * 8 + "i" * 48) is not None


def test_workspace_hands_out_views_of_one_buffer():
    ws = Workspace("cpu")
    a = ws.get("x", (2, 3), torch.float32)
    assert ws.get("x", (2, 3), torch.float32) is a and ws.get("x", [2, 3], torch.float32).shape == (2, 3)
    b = ws.get("x", (3, 2), torch.float32)
    assert b.shape == (3, 2) and b.data_ptr() == a.data_ptr()
    assert ws.get("x", (2, 3), torch.bfloat16).dtype == torch.bfloat16
    with torch.inference_mode():
        c = ws.get("x", (3, 2), torch.float32)
        assert c.data_ptr() == b.data_ptr()
    ws.get("x", (3, 2), torch.float32).add_(1)
    big = ws.get("x", (40, 2), torch.float32)
    with torch.inference_mode():
        assert ws.get("x", (3, 2), torch.float32).data_ptr() == big.data_ptr()
