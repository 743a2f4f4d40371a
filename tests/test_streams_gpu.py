"""Steps whose kernels may start before the one in front of them has ended
(programmatic dependent launch): every order of steps with the calls that read or
write the same memory gives the bits of the same calls waited for one by one."""
import numpy as np
import pytest

import freelb_b200 as F
from freelb_b200 import geometry

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


def shaped(storage, model, ni, shape):
    lat = F.cavity(ni, tau=0.55, storage=storage, model=model)
    lat.set_launch(*shape)
    return lat


def blocks(storage, model):
    """A cavity of 98^3 in blocks with halos, in the shape the library picks."""
    ni = 96
    parts = geometry.uneven_blocks(ni, edges=(32, 48), seed=1)
    lat = F.Lattice.blocks(geometry.block_tuples(parts), 0.55, mode="halo", storage=storage,
                           model=model)
    flags = F.cavity_flags(ni)
    u = np.zeros((flags.size, 3))
    u[flags == 8, 0] = 0.1
    for k, b in enumerate(parts):
        lat.upload_flags(geometry.slice_block(flags, ni + 2, b), block=k)
        lat.upload_field("u", geometry.slice_block(u, ni + 2, b, comps=3), block=k)
    return lat


WIDE, PERSISTENT, PIPELINE = (2, 0, 4), (4, 8, 2), (4, -1, 4)


@pytest.mark.parametrize("make", [
    lambda: shaped("fp32", "bgk", 148, WIDE), lambda: shaped("fp32", "mrt", 148, (4, 0, 2)),
    lambda: shaped("fp32", "les", 126, PERSISTENT), lambda: shaped("fp32s", "bgk", 126, (4, 0, 2)),
    lambda: shaped("fp64", "bgk", 126, (4, 0, 2)), lambda: shaped("fp16s", "bgk", 148, WIDE),
    lambda: shaped("fp16s", "mrt", 126, (4, 0, 2)), lambda: shaped("fp16s", "bgk", 126, PIPELINE),
    lambda: shaped("fp16s", "les", 148, PIPELINE), lambda: blocks("fp32", "bgk"),
    lambda: blocks("fp16s", "bgk"), lambda: blocks("fp64", "bgk"), lambda: blocks("fp32s", "bgk"),
])
def test_every_step_kernel_keeps_its_order(gpu_ok, make):
    """Each form of the step that may start early, on lattices of several waves of
    CTAs, and the halo copies after it: 24 steps in a row against 24 waited for."""
    import torch
    out = []
    for wait in (False, True):
        lat = make()
        torch.cuda.synchronize()
        if wait:
            for _ in range(24):
                lat.step(1)
                torch.cuda.synchronize()
        else:
            lat.step(24)
        out.append([lat.download_pops(block=b) for b in range(lat.nblocks)])
        lat.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def test_a_reported_error_does_not_fail_the_next_call(gpu_ok):
    """A download on a stream that is being captured is an error, once."""
    import torch
    from cuda.bindings import runtime as rt
    lat = F.cavity(20)
    lat.step(3)
    want = lat.download_pops()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    mode = rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal
    assert rt.cudaStreamBeginCapture(stream.cuda_stream, mode)[0] == 0
    with pytest.raises(F.FlbError):
        lat.download_pops(stream=stream)
    rt.cudaStreamEndCapture(stream.cuda_stream)
    rt.cudaGetLastError()
    assert np.array_equal(lat.download_pops(stream=stream), want)
