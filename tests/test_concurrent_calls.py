"""One-launch forms, chained launches and a tile queue on four streams at once, from four
threads: every result is that of the call alone."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _calls():
    """name -> (fields, call on copies of them)."""
    import torch

    from npbench_gb300 import stencils
    gen = torch.Generator(device="cuda")
    gen.manual_seed(12)

    def r(*shape, dtype=torch.float64, size=1.0):
        return size * torch.rand(shape, generator=gen, device="cuda", dtype=dtype)

    f32 = torch.float32
    flow = 2 / 59, 2 / 59, 1e-5

    def cavity(u, v, p):
        stencils.cavity_flow(60, 60, 4, 6, u, v, flow[2], flow[0], flow[1], p, 1.0, 0.1)

    def channel(u, v, p):
        stencils.channel_flow(6, u, v, flow[2], flow[0], flow[1], p, 1.0, 0.1, 1e-9)

    return {
        "bands": ([r(300, 500, dtype=f32), r(300, 500, dtype=f32)], lambda a, b: stencils.jacobi_2d_kernel(30, a, b)),
        "wide bands": ([r(450, 2050, dtype=f32), r(450, 2050, dtype=f32)],
                       lambda a, b: stencils.jacobi_2d_kernel(20, a, b)),
        "loop": ([r(300, 400), r(300, 400)], lambda a, b: stencils.jacobi_2d_kernel(20, a, b)),
        "strips": ([r(200, 700), r(200, 700)], lambda a, b: stencils.jacobi_2d_kernel(10, a, b)),
        "resident": ([r(20000, dtype=f32), r(20000, dtype=f32)], lambda a, b: stencils.jacobi_1d_kernel(100, a, b)),
        "heat": ([r(40, 50, 60), r(40, 50, 60)], lambda a, b: stencils.heat_3d_kernel(6, a, b)),
        "cavity": ([r(60, 60, size=1e-3) for _ in range(3)], cavity),
        "channel": ([r(60, 60, size=1e-3) for _ in range(3)], channel),
    }


@pytest.mark.parametrize("queue", [False, True])
def test_results_do_not_depend_on_what_else_runs(queue):
    import torch

    from npbench_gb300 import _lib
    from npbench_gb300.queue import TileQueue
    calls = _calls()
    want = {}
    for name, (fields, call) in calls.items():
        want[name] = [x.clone() for x in fields]
        call(*want[name])
    torch.cuda.synchronize()
    wrong, errors = [], []

    def work(n):
        try:
            names = sorted(calls)
            with torch.cuda.stream(torch.cuda.Stream()):
                for k in range(48):
                    name = names[(k * (2 * n + 1) + n) % len(names)]
                    got = [x.clone() for x in calls[name][0]]
                    calls[name][1](*got)
                    if not all(torch.equal(a, b) for a, b in zip(got, want[name])):
                        wrong.append(name)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(n,)) for n in range(4)]
    if queue:
        grids = [[torch.rand((50 + n, 60), device="cuda", dtype=torch.float64) for _ in range(2)] for n in range(3)]
        with TileQueue(max_slots=4, ctas_per_sm=1) as q:
            stream = torch.cuda.Stream()
            for t in threads:
                t.start()
            for a, b in grids:
                q.submit(a, b, 2000)
                q.kick(stream)
            for t in threads:
                t.join()
            stream.synchronize()
    else:
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    torch.cuda.synchronize()
    _lib.device_status()
    assert not errors and not wrong
