"""Several host threads in the library at once, each on its own stream: launches with different
amounts of shared memory."""

import threading

import pytest
import torch

from gmaster_b200 import _lib, sht
from gmaster_b200.workspaces import LUFactor

pytestmark = pytest.mark.gpu


def _run(jobs, reps):
    errors = []

    def work(job):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(reps):
                    job()
                torch.cuda.current_stream().synchronize()
        except Exception as err:   # noqa: BLE001 - reported by the test
            errors.append(err)

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_ring_stages_of_different_sizes(cuda):
    """Every length class of the ring kernels has its own shared-memory size; plans and scratch are
    made before, so that the threads only launch."""
    jobs, wants = [], []
    for nside in (32, 512, 256, 1024):
        plan = sht.get_plan(nside, 2 * nside)
        maps = torch.randn((1, plan.npix), dtype=torch.float64, device="cuda")
        syn = torch.randn((plan.L, plan.nlanes, 1, 4), device="cuda")
        sht.ring_synthesis(plan, syn, _lib.MIXED)
        want = sht.ring_analysis(plan, maps, _lib.MIXED)
        got = torch.zeros_like(want)
        wants.append((got, want))

        def job(plan=plan, maps=maps, syn=syn, got=got):
            sht.ring_analysis(plan, maps, _lib.MIXED, out=got)
            sht.ring_synthesis(plan, syn, _lib.MIXED)

        jobs.append(job)
    torch.cuda.synchronize()
    _run(jobs, 150)
    for got, want in wants:
        assert torch.equal(got, want)


def test_lu_solves_of_different_sizes(cuda):
    jobs = []
    for n in (40, 159, 900, 3000):
        lu = LUFactor(torch.eye(n, dtype=torch.float64, device="cuda") * 2)
        rhs = {r: torch.randn((n, r), dtype=torch.float64, device="cuda") for r in (1, 300)}

        def job(lu=lu, rhs=rhs, n=n):
            for b in rhs.values():
                lu.solve(b)
            if n <= 900:
                LUFactor(torch.eye(n, dtype=torch.float64, device="cuda"))

        jobs.append(job)
    torch.cuda.synchronize()
    _run(jobs, 60)
