"""The tile kernels' own source on the CPU (schedules/emulator.cpp), every warp, copy and group of products in random order: what the source does not order shows as
other bits, a barrier that a warp reaches twice in one turn is counted, and a block in which a wait runs out still comes to its end."""
import ctypes as C
import importlib
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

from conftest import ROOT

CSRC = ROOT / "dhammic-ai_b200" / "csrc"
_PTR = ("x", "B", "C", "y", "dy", "dx", "dB", "dC", "states", "dstates", "tcum", "dtT", "skipT", "D", "seed", "out_state", "ysq", "g_", "ddtx", "dyx", "gS", "status", "extreme")


class Args(C.Structure):
    _fields_ = ([(k, C.c_int) for k in "bThgpn"] + [(k, C.c_void_p) for k in _PTR] + [(k, C.c_int) for k in ("flags", "whole", "np")] + [("cut", C.c_int * 5), ("ctas", C.c_int)]
                + [("schedule", C.c_uint)] + [(k, C.c_int) for k in ("in_order", "expire", "lose_copy", "overruns", "underflows", "hung", "expiries")])


@pytest.fixture(scope="session")
def emulator(tmp_path_factory):
    out = tmp_path_factory.mktemp("schedules")
    for f in CSRC.glob("ssd_tc*.cuh"):
        (out / f.name).write_text(f.read_text().replace("extern __shared__", "extern"))
    for name in ("ssd_common.cuh", "ssd_cumsum.cuh", "ssd_ptx.cuh"):  # the emulator's own
        (out / name).write_text("#pragma once\n")
    cuda = Path(importlib.import_module("dhammic-ai_b200.build")._nvcc()).resolve().parent.parent / "include"
    lib = out / "emulator.so"
    subprocess.run(["g++", "-O2", "-fno-strict-aliasing", "-std=c++17", "-fPIC", "-shared", "-w", f"-I{cuda}", f"-I{out}", str(ROOT / "tests" / "schedules" / "emulator.cpp"), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


def bf16(t):
    return t.bfloat16().view(torch.int16).numpy().copy()


def wide(a):
    return torch.from_numpy(a.copy()).view(torch.bfloat16).double()


class Call:
    """One launch's tensors, and what it leaves."""
    def __init__(self, T, h, g, skip=True, scaled=True, b=1, p=64, n=128, whole=0, cut=(), ctas=1):
        gen = torch.Generator().manual_seed(T + 7 * h)
        nt = (T + 127) // 128
        r = lambda *s: torch.randn(*s, generator=gen)
        self.t = {"x": bf16(r(b, T, h, p)), "B": bf16(r(b, T, g, n) / 11), "C": bf16(r(b, T, g, n)), "dy": bf16(r(b, T, h, p)), "y": bf16(torch.zeros(b, T, h, p)),
                  "dx": bf16(torch.zeros(b, T, h, p)), "dB": bf16(torch.zeros(b, T, g, n)), "dC": bf16(torch.zeros(b, T, g, n)),
                  "states": bf16(r(b * nt * h * 128, 64)), "dstates": bf16(r(b * nt * h * 128, 64))}
        a = torch.zeros(b, h, nt * 128)
        a[..., :T] = -0.05 * torch.rand(b, h, T, generator=gen)
        f = {"tcum": a.view(b, h, nt, 128).cumsum(-1), "D": r(h), "seed": r(b, h, p, n), "out_state": torch.zeros(b, h, p, n), "ysq": torch.zeros(b, nt, h, 2, 128),
             "g_": torch.zeros(b, h, nt * 128), "ddtx": torch.zeros(b, h, nt * 128), "dyx": torch.zeros(b, h, nt * 128), "gS": torch.zeros(b, h, nt, 8)}
        if scaled:
            f["dtT"] = torch.rand(b, h, nt * 128, generator=gen)
        if skip:
            f["skipT"] = r(b, h, nt * 128)
        self.t.update({k: np.ascontiguousarray(v.numpy(), dtype=np.float32) for k, v in f.items()})
        self.t.update(status=np.zeros(1, np.int32), extreme=np.zeros(1, np.int32))
        self.first = {k: v.copy() for k, v in self.t.items()}
        self.args = Args(b=b, T=T, h=h, g=g, p=p, n=n, flags=1, whole=whole, np=max(1, len(cut) - 1), ctas=ctas, **{k: self.t[k].ctypes.data for k in _PTR if k in self.t})
        for i, c in enumerate(cut):
            self.args.cut[i] = c

    def run(self, kernel, *more, schedule=0, in_order=0, expire=0, lose_copy=-1):
        for k, v in self.t.items():
            v[...] = self.first[k]
        for k, v in (("schedule", schedule), ("in_order", in_order), ("expire", expire), ("lose_copy", lose_copy)):
            setattr(self.args, k, v)
        kernel(C.byref(self.args), *more)
        return {k: v.copy() for k, v in self.t.items()}


CASES = [  # kernel, its own arguments, tensors
    ("forward", (), dict(T=128, h=1, g=1)),
    ("forward", (), dict(T=300, h=1, g=1, skip=False)),
    ("forward", (), dict(T=640, h=1, g=1, scaled=False)),
    ("forward", (), dict(T=768, h=2, g=1, whole=1, cut=(0, 3, 6))),
    ("forward", (), dict(T=768, h=1, g=1, cut=(0, 1, 3, 6))),
    ("states", (), dict(T=640, h=1, g=1)),
    ("reverse", (1,), dict(T=896, h=1, g=1)),
    ("reverse", (2,), dict(T=640, h=2, g=1)),
    ("summary", (1, 0), dict(T=768, h=1, g=1)),
    ("summary", (2, 1), dict(T=640, h=2, g=1)),
    ("backward", (), dict(T=256, h=1, g=1, skip=False)),
    ("backward", (), dict(T=384, h=2, g=2)),
    ("backward", (), dict(T=256, h=2, g=1)),
    ("backward", (), dict(T=200, h=3, g=1, scaled=False)),
]
IDS = [f"{k}{''.join(map(str, m))}-{kw['T']}-{kw['h']}-{kw['g']}" for k, m, kw in CASES]


@pytest.mark.parametrize("kernel,more,shape", CASES, ids=IDS)
def test_any_order_gives_the_same_bits(emulator, kernel, more, shape):
    call, f = Call(**shape), getattr(emulator, kernel)
    want = call.run(f, *more, in_order=1)
    assert call.args.hung == call.args.overruns == call.args.underflows == 0 and want["status"][0] == 0
    for schedule in range(1, 13):
        got = call.run(f, *more, schedule=schedule)
        assert (call.args.hung, call.args.overruns, call.args.underflows) == (0, 0, 0), schedule
        for k, v in want.items():
            assert np.array_equal(v.view(np.uint8), got[k].view(np.uint8)), (schedule, k)


@pytest.mark.parametrize("kernel,more,shape", CASES, ids=IDS)
def test_a_wait_that_runs_out_ends_the_block(emulator, kernel, more, shape):
    """Waits given up at random, or because a copy never lands: the block reports it and comes to its end, and no warp is counted twice in one turn of a barrier."""
    call, f, expiries = Call(**shape), getattr(emulator, kernel), 0
    for schedule in range(1, 25):
        how = dict(expire=1) if schedule % 2 else dict(lose_copy=schedule // 2 - 1)
        got = call.run(f, *more, schedule=schedule, **how)
        assert (call.args.hung, call.args.overruns) == (0, 0), schedule
        assert int(got["status"][0]) == int(call.args.expiries > 0), schedule
        expiries += call.args.expiries
    assert expiries > 0


@pytest.mark.parametrize("tiles,h,whole,cut", [(4, 1, 0, (0, 2, 4)), (7, 2, 1, (0, 4, 7)), (8, 3, 1, (0, 3, 6, 8)), (9, 2, 0, (0, 3, 5, 7, 9))])
def test_cut_walks_have_the_bits_of_whole_ones(emulator, tiles, h, whole, cut):
    shape = dict(T=128 * tiles - 50, h=h, g=1)
    want, got = (Call(**shape, **kw).run(emulator.forward, schedule=3) for kw in ({}, dict(whole=whole, cut=cut)))
    for k in ("y", "states", "out_state", "ysq"):
        assert np.array_equal(want[k].view(np.uint8), got[k].view(np.uint8)), k


def test_emulated_walk_is_the_scan(emulator):
    """Against the recurrence in 64 bits, whose operands the kernel rounds to bf16."""
    call = Call(T=300, h=2, g=1)
    got = call.run(emulator.forward, in_order=1)
    t = {k: torch.from_numpy(v) for k, v in call.first.items()}
    x, B, Cm = (wide(call.first[k])[0] for k in ("x", "B", "C"))
    for h in range(2):
        H, y = t["seed"][0, h].double(), []
        cum = t["tcum"][0, h].reshape(-1).double()
        for i in range(300):
            a = cum[i] - (cum[i - 1] if i % 128 else 0.0)
            H = 2.0 ** a * H + t["dtT"][0, h, i].double() * x[i, h].unsqueeze(1) * B[i, 0]
            y.append(H @ Cm[i, 0] + t["skipT"][0, h, i].double() * x[i, h])
        y = torch.stack(y)
        assert float((wide(got["y"])[0, :, h] - y).abs().max() / y.abs().max()) < 2e-2
        assert float((torch.from_numpy(got["out_state"])[0, h].double() - H).abs().max() / H.abs().max()) < 1e-2
