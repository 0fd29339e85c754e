"""One context used by several threads at once: its stage functions share the context's
scratch block and take turns on it, whatever sizes the others ask for."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_of_one_context_take_turns_on_its_scratch(gpu):
    import torch
    from simcraft_b200 import fluid
    from simcraft_b200._capi import lib
    from simcraft_b200.solver import Context

    dims, h = (17, 12, 21), 1 / 16
    ptr = lambda a: ctypes.c_void_p(a.data_ptr())
    ctx = Context(0)  # calls below stay on its own stream
    threads, rounds = 4, 12
    jobs, errors = [], []
    for k in range(threads):
        mine = []
        for i in range(rounds):
            n = (1, 4097, 300, 60000, 31, 20000)[(i + k) % 6]
            rng = np.random.default_rng(100 * k + i)
            pos = torch.from_numpy(rng.uniform(0, 1, (n, 3)) * np.array(dims) * h).cuda()
            vel = torch.from_numpy(rng.normal(size=(n, 3))).cuda()
            a = fluid.p2g(pos, vel, dims, h, context=Context(0))
            grids = [a[g] for g in ("u", "v", "w", "ulast", "vlast", "wlast")]
            want = fluid.g2p(pos, vel, dims, h, *grids, context=Context(0))
            mine.append((pos, vel, grids, want, vel.clone()))
        jobs.append(mine)
    torch.cuda.synchronize()

    def work(mine):
        for pos, _, grids, _, out in mine:
            rc = lib().sc_flip_g2p_device(ctx.handle, pos.shape[0], ptr(pos), ptr(out), *dims, h, *[ptr(g) for g in grids], 0.97)
            if rc:
                errors.append(rc)

    pool = [threading.Thread(target=work, args=(m,)) for m in jobs]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    ctx.synchronize()
    assert not errors
    for mine in jobs:
        for _, _, _, want, out in mine:
            assert torch.equal(out, want)
