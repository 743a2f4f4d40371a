"""Steps whose kernels may start before the one in front of them has ended
(programmatic dependent launch): every order of steps with the calls that read or
write the same memory gives the bits of the same calls waited for one by one."""
import numpy as np
import pytest

import freelb_b200 as F

pytestmark = pytest.mark.gpu


def halfway_lattice(storage, ni=20):
    n = ni + 2
    lat = F.Lattice(n, n, n, 0.6, storage=storage, tasks=((2 | 4 | 8, "bulk"),))
    lat.upload_flags(F.cavity_flags(ni))
    u = np.zeros((n ** 3, 3))
    u[F.cavity_flags(ni) == 8, 0] = 0.1
    lat.upload_field("u", u)
    return lat, [F.BounceBackManager(lat, 4, 1, kind="normal"),
                 F.BounceBackManager(lat, 8, 1, kind="movingwall")]


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64", "fp32s"])
@pytest.mark.parametrize("own_stream", [False, True])
def test_steps_and_managers_keep_their_order(gpu_ok, storage, own_stream):
    import torch
    out = []
    for wait in (False, True):
        stream = torch.cuda.Stream() if own_stream else None
        lat, walls = halfway_lattice(storage)
        sync = torch.cuda.synchronize if wait else (lambda: None)
        torch.cuda.synchronize()
        rhos = []
        for k in range(30):
            lat.step(1 + k % 3, stream)
            sync()
            for wall in walls:
                wall.apply(stream)
                sync()
            if k % 10 == 9:
                lat.compute_rhou(6, stream)
                sync()
                rhos.append(lat.download_field("rho", stream=stream))
        out.append((lat.download_pops(stream=stream), rhos))
    assert np.array_equal(out[0][0], out[1][0])
    assert all(np.array_equal(a, b) for a, b in zip(out[0][1], out[1][1]))


@pytest.mark.parametrize("storage", ["fp32", "fp16s"])
def test_steps_captured_by_the_caller(gpu_ok, storage):
    import torch
    a, b = (F.cavity(24, tau=0.55, storage=storage) for _ in range(2))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    a.step(2, stream)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        a.step(2, stream)
    for _ in range(4):
        graph.replay()
    torch.cuda.synchronize()
    b.step(10)
    assert np.array_equal(a.download_pops(), b.download_pops())
