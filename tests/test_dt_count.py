"""hp_dt_noalloc's counters of finished blocks: a call is right whatever the
calls before it left in the counter it shares with them (csrc/hp_dt_count.h,
on the CPU), and a captured call, which is replayed many times, gives the time
step of the state in its buffers at each replay, beside eager calls that take
every counter."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from hydraphase import cases, lib

HERE = os.path.dirname(os.path.abspath(__file__))


def test_calls_after_an_overlap_count_right(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "dt_count_check.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    mixed, wrong = map(int, re.search(r"mixed (\d+), later calls wrong (\d+)", out.stdout).groups())
    assert mixed > 100 and wrong == 0 and out.returncode == 0, out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 257, 100_000])
def test_captured_call_replays(n):
    import torch
    sp = cases.shock_bubble(n=23, alpha_min=0.1)
    rng = np.random.default_rng(3)
    pick = rng.integers(0, sp.cu.shape[1], n)
    states = [torch.from_numpy(np.ascontiguousarray(sp.cu[:, pick] * (1.0 + 0.1 * k))).cuda() for k in range(3)]
    dl = torch.from_numpy(rng.uniform(0.01, 0.02, n)).cuda()
    p = sp.params(cfl=0.3)

    def call(cn, out):
        assert lib().hp_dt_noalloc(cn.data_ptr(), n, dl.data_ptr(), n, ctypes.byref(p), out.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream) == 0

    ref = torch.zeros(3, dtype=torch.float64, device="cuda")
    for k in range(3):
        call(states[k], ref[k:])
    buf, out = states[0].clone(), torch.zeros(1, dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(buf, out)
    other = torch.zeros(1, dtype=torch.float64, device="cuda")
    got = []
    for k in (1, 2, 0, 1):
        buf.copy_(states[k])
        out.fill_(-1.0)
        graph.replay()
        got.append(out.clone())
        for _ in range(1025):
            call(states[k], other)
        assert other.item() == ref[k].item()
    assert [g.item() for g in got] == [ref[k].item() for k in (1, 2, 0, 1)]
    assert (ref > 0).all()
