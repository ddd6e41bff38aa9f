"""Calls on another stream while a tile queue's worker holds a part of every SM: they must not
wait for the worker to end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fields(*shape, n=2, dtype="float32"):
    import torch
    return [1e-3 * torch.rand(shape, device="cuda", dtype=getattr(torch, dtype)) for _ in range(n)]


def _calls():
    from npbench_gb300 import stencils

    def jacobi(shape, dtype):
        A, B = _fields(*shape, dtype=dtype)
        return lambda: stencils.jacobi_2d_kernel(20, A, B)

    def cavity(ny, nx):
        u, v, p = _fields(ny, nx, n=3, dtype="float64")
        return lambda: stencils.cavity_flow(nx, ny, 3, 5, u, v, 1e-5, 2 / (nx - 1), 2 / (ny - 1), p, 1.0, 0.1)

    def jacobi_1d():
        A, B = _fields(32000)
        return lambda: stencils.jacobi_1d_kernel(200, A, B)

    return {"jacobi_2d f32 300x300": lambda: jacobi((300, 300), "float32"),
            "jacobi_2d f32 1403x1177": lambda: jacobi((1403, 1177), "float32"),
            "jacobi_2d f64 301x481": lambda: jacobi((301, 481), "float64"),
            "jacobi_2d f64 1000x1000": lambda: jacobi((1000, 1000), "float64"),
            "cavity 101x101": lambda: cavity(101, 101), "cavity 201x201": lambda: cavity(201, 201),
            "cavity 330x200": lambda: cavity(330, 200), "cavity 100x500": lambda: cavity(100, 500),
            "jacobi_1d f32": jacobi_1d}


@pytest.mark.parametrize("name", ["jacobi_2d f32 300x300", "jacobi_2d f32 1403x1177", "jacobi_2d f64 301x481",
                                  "jacobi_2d f64 1000x1000", "cavity 101x101", "cavity 201x201", "cavity 330x200",
                                  "cavity 100x500", "jacobi_1d f32"])
def test_a_call_does_not_wait_for_the_worker(name):
    import torch

    from npbench_gb300 import _lib
    from npbench_gb300.queue import TileQueue
    call = _calls()[name]()
    small = torch.rand((60, 60), device="cuda", dtype=torch.float64), torch.rand((60, 60), device="cuda",
                                                                                 dtype=torch.float64)
    torch.cuda.synchronize()
    work, other = torch.cuda.Stream(), torch.cuda.Stream()
    with TileQueue(max_slots=4, ctas_per_sm=1) as q:  # the serving loop's worker
        call()  # loads its kernels, which a running one would delay
        torch.cuda.synchronize()
        slot = q.submit(*small, 10000)  # 0.4 s
        q.kick(work)
        with torch.cuda.stream(other):
            call()
        other.synchronize()
        assert slot not in q.poll() and q.state()["running"]
        work.synchronize()
        assert slot in q.poll()
    _lib.device_status()


def test_one_launch_forms_return_when_the_queue_has_gone():
    import torch

    from npbench_gb300 import _lib, stencils
    from npbench_gb300.queue import TileQueue

    def launches():
        A, B = _fields(300, 300)
        n0 = _lib.launches()
        stencils.jacobi_2d_kernel(20, A, B)
        torch.cuda.synchronize()
        return _lib.launches() - n0

    assert launches() == 1
    q = TileQueue(max_slots=2)
    assert launches() == 38
    q.destroy()
    assert launches() == 1
