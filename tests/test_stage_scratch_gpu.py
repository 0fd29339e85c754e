"""Scratch of the stage functions: a context's own memory, kept between calls.

Calls of growing and shrinking sizes, on changing streams, from several threads
with a context each, and with the context destroyed right after the call, give
the bits that a fresh context gives."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 4097, 300, 60000, 0, 60000, 31]


@pytest.fixture(scope="module")
def torch_mod(gpu):
    import torch
    return torch


def _scene(torch, n, dims, h, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0, 1, (n, 3)) * np.array(dims) * h
    return torch.from_numpy(pos).cuda(), torch.from_numpy(rng.normal(size=(n, 3))).cuda()


def _once(fluid, pos, vel, dims, h, ctx):
    a = fluid.p2g(pos, vel, dims, h, context=ctx)
    out = [a[k] for k in ("u", "v", "w", "uw", "uvalid")]
    if pos.shape[0]:
        out.append(fluid.g2p(pos, vel, dims, h, a["u"], a["v"], a["w"], a["ulast"], a["vlast"], a["wlast"], context=ctx))
    return out


@pytest.mark.parametrize("threads", [1, 3])
def test_reused_scratch_gives_a_fresh_contexts_bits(torch_mod, threads):
    from simcraft_b200 import fluid
    from simcraft_b200.solver import Context
    t = torch_mod
    dims, h = (17, 12, 21), 1 / 16
    scenes = [_scene(t, n, dims, h, i) for i, n in enumerate(SIZES)]
    want = [_once(fluid, p, v, dims, h, Context(0)) for p, v in scenes]  # destroyed right after its calls
    t.cuda.synchronize()
    got, errors = [[] for _ in range(threads)], []

    def work(k):
        try:
            ctx = Context(0)
            streams = [t.cuda.Stream(), t.cuda.Stream()]
            for i, (p, v) in enumerate(scenes):
                s = streams[(i // 2) & 1]
                with t.cuda.stream(s):
                    got[k].append(_once(fluid, p, v, dims, h, ctx))
            t.cuda.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    pool = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for th in pool:
        th.start()
    for th in pool:
        th.join()
    assert not errors
    for k in range(threads):
        for a, b in zip(want, got[k]):
            for x, y in zip(a, b):
                assert t.equal(x, y)
