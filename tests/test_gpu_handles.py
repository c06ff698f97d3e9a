"""Handles are independent of one another (needs a B200): host threads with
handles whose kernels use different amounts of shared memory."""
import dataclasses
import threading

import numpy as np
import pytest

import nbk
from helpers import ALL, PARAMS, mixed_box, wider_lj

pytestmark = pytest.mark.gpu


class _Caller:
    """One handle on a stream of its own: an evaluation, an adjoint and a patch
    sort, and what the three return."""

    def __init__(self, p, beta, types, max_patch):
        import torch
        self.torch = torch
        self.p, system = p, p.system
        lj = wider_lj(system.lj_table(), types)
        self.stream = torch.cuda.Stream()
        self.s = self.stream.cuda_stream
        self.nb = nbk.Nonbonded(dataclasses.replace(PARAMS, ewaldcof=beta), lj)
        self.nb.setup(p, stream=self.s)
        n = p.atomStorageSize
        self.xyzq = torch.from_numpy(p.xyzq.copy()).cuda()
        rng = np.random.default_rng(5)
        self.w = torch.from_numpy(rng.standard_normal((n, 4)).astype(np.float32)).cuda()
        self.X = torch.zeros((6, n), dtype=torch.int64, device="cuda")
        self.g = torch.zeros((n, 4), device="cuda")
        self.G = torch.zeros((4, n), dtype=torch.int64, device="cuda")
        self.gab = torch.zeros(2 * types * types, dtype=torch.float64, device="cuda")
        self.layout = nbk.ResidentLayout(system, p, shuffle_seed=1)
        self.order = torch.zeros(len(self.layout.ids), dtype=torch.int32, device="cuda")
        self.max_patch = max_patch
        torch.cuda.synchronize()
        self.nb.build_tile_lists(p, xyzq=self.xyzq, stream=self.s)
        self.nb.force(p, ALL | nbk.NBK_PAIRLIST, xyzq=self.xyzq, stream=self.s)

    def call(self):
        self.nb.force(self.p, ALL, xyzq=self.xyzq, d_fixed=self.X, stream=self.s)
        for _ in range(4):
            self.nb.adjoint(self.w, self.w, 0.1, 0.1, 0.1, self.g, self.gab, grad_fixed=self.G, stream=self.s)
            self.layout.sort_patch_atoms(self.order, max_patch_atoms=self.max_patch, stream=self.s)

    def result(self):
        self.stream.synchronize()
        return [t.cpu().numpy().copy() for t in (self.X, self.G, self.order)]


# Few LJ types, short tables and small patches in half of the threads; 100 types,
# longer tables and the largest patches in the others. Each kernel's shared-memory
# limit has to hold for all, whoever launched last.
def test_threads_with_different_shared_memory():
    p = nbk.Packed(mixed_box(seed=12, natoms=3001))
    callers = [_Caller(p, 0.2579, 34, 512) if k % 2 else _Caller(p, 0.6, 100, 2000) for k in range(8)]
    want = []
    for c in callers:
        c.call()
        want.append(c.result())
    failed = []

    def work(c):
        try:
            for _ in range(300):
                c.call()
        except nbk.NbkError as e:
            failed.append(str(e))

    threads = [threading.Thread(target=work, args=(c,)) for c in callers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    got = [c.result() for c in callers]
    assert not failed, failed
    for a, b in zip(want, got):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
