"""Host operands in pageable memory: pieces around the pinned slots of 1 MB, more of them than
there are slots, rows with gaps, pinned memory beside pageable memory, several threads at
once, and a call that fails after others succeeded.  Integer results are exact."""
import threading

import numpy as np
import pytest
import torch

import cpu_ops_b200 as c
from cpu_ops_b200 import _capi

pytestmark = pytest.mark.gpu


def problem(m, n, k, pad, seed, pinned=()):
    g = torch.Generator().manual_seed(seed)
    t = {"A": torch.randint(0, 256, (m, k + pad), dtype=torch.uint8, generator=g),
         "B": torch.randint(-128, 128, (k, n + pad), dtype=torch.int8, generator=g),
         "C": torch.randint(-1000, 1001, (m, n + pad), dtype=torch.int32, generator=g),
         "D": torch.full((m, n + pad), 77, dtype=torch.int32)}
    t = {name: x.pin_memory() if name in pinned else x for name, x in t.items()}
    # |sums| < 2^53: exact in f64
    want = (t["A"][:, :k].cuda().double() @ t["B"][:, :n].cuda().double()).to(torch.int32).cpu() + t["C"][:, :n]
    return t, want


def run(t, m, n, k, pad):
    op = c.GemmU8S8S32()
    x = {name: v.numpy() for name, v in t.items()}
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.TensorRef(x["A"], k + pad), c.TensorRef(x["B"], n + pad),
                         c.TensorRef(x["C"], n + pad), c.TensorRef(x["D"], n + pad), c.LinearCombination(1, 1)))
    assert st == c.Status.kSuccess, _capi.last_error()


def check(t, want, n):
    assert torch.equal(t["D"][:, :n], want)
    assert bool((t["D"][:, n:] == 77).all())


# 262144 words a slot: one slot less a row, exactly one, one more; 2300 x 2400 words are 22 slots
@pytest.mark.parametrize("m,n,k,pad,pinned", [
    (255, 1024, 300, 0, ()), (256, 1024, 300, 0, ()), (257, 1024, 300, 0, ()), (128, 128, 64, 0, ()), (100, 163, 200, 1, ()),
    (300, 1000, 700, 3, ()), (1100, 1027, 513, 0, ()), (2300, 2400, 1024, 3, ()), (1024, 1024, 1024, 0, ("A",)),
    (1024, 1024, 1024, 0, ("D",)), (1024, 1024, 1024, 3, ("A", "B", "C", "D"))])
def test_pageable(gpu, m, n, k, pad, pinned):
    t, want = problem(m, n, k, pad, m + n, pinned)
    run(t, m, n, k, pad)
    check(t, want, n)


def test_threads(gpu):
    jobs = [(problem(1100 + 64 * i, 900, 512, i, i), 1100 + 64 * i, i) for i in range(4)]
    errors = []

    def work(job):
        (t, want), m, pad = job
        try:
            for _ in range(5):
                t["D"].fill_(77)
                run(t, m, 900, 512, pad)
                check(t, want, 900)
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors[0]


def test_a_refused_call_writes_nothing(gpu):
    t, want = problem(1200, 800, 256, 0, 9)
    x = {name: v.numpy() for name, v in t.items()}
    op = c.GemmU8S8S32(asynchronous=True)  # host operands cannot be asynchronous
    st = op(op.Arguments(c.GemmCoord(1200, 800, 256), c.TensorRef(x["A"], 256), c.TensorRef(x["B"], 800),
                         c.TensorRef(x["C"], 800), c.TensorRef(x["D"], 800), c.LinearCombination(1, 1)))
    assert st != c.Status.kSuccess
    assert bool((t["D"] == 77).all())
    run(t, 1200, 800, 256, 0)
    check(t, want, 800)
