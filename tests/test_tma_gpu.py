"""The FP16S bulk-copy kernel (k_pull_tma, launch ctas_per_sm = -2 / -3): the
sources of each tile are staged in shared memory by bulk asynchronous copies
and collided there.  It must give the direct kernel's bits on every cell, for
every model, on lattices whose tiles fall across row ends, padding and the
unstaged tiles near the first and last planes; its bounded waits must report a
wait that gave up through flb_device_status, and leave the handle usable."""
import ctypes

import numpy as np
import pytest

import freelb_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def pair(make, steps, mode, rounding="default"):
    """The same lattice stepped by the direct kernel and by the bulk-copy kernel."""
    a, b = make(), make()
    a.set_rounding(rounding)
    b.set_rounding(rounding)
    a.set_launch(1, 0, 4)
    b.set_launch(4, mode, 4)
    a.step(steps)
    b.step(steps)
    b.device_status()
    return a, b


@pytest.mark.parametrize("rounding", ["nearest", "stochastic"])
@pytest.mark.parametrize("mode", [-2, -3])
@pytest.mark.parametrize("model", ["bgk", "mrt", "les"])
@pytest.mark.parametrize("ni", [22, 30, 62])
def test_tma_equals_direct_kernel_on_cavity(gpu_ok, model, ni, mode, rounding):
    a, b = pair(lambda: F.cavity(ni, tau=0.55, storage="fp16s", model=model), 25, mode,
                rounding)
    assert np.array_equal(a.download_pops(), b.download_pops())


@pytest.mark.parametrize("model", ["bgk", "mrt", "les"])
@pytest.mark.parametrize("dims", [(23, 11, 40), (24, 30, 19), (40, 9, 30), (31, 17, 25)])
def test_tma_equals_direct_kernel_on_random_flags(gpu_ok, model, dims):
    """Every op and flag value (random first-match task list), perturbed
    populations and fields; pitch - nx from 0 to 1 (rows ending right before
    the next row or one half short of it)."""
    nx, ny, nz = dims
    N = nx * ny * nz
    rng = np.random.default_rng(nx + 7 * ny + 31 * nz)
    flags = rng.choice(np.array([1, 2, 4, 8, 16, 2 | 16, 32], dtype=np.uint8), size=N,
                       p=[.1, .5, .1, .1, .1, .05, .05])
    tasks = ((2, "bulk"), (4, "bounceback"), (8, "movingwall"), (16, "field_bgk"))
    w = np.repeat(O.W, N)
    pops = (w * (1 + 0.05 * rng.standard_normal(19 * N))).astype(np.float32)
    rho = (1 + 0.01 * rng.standard_normal(N)).astype(np.float32)
    u = (0.03 * rng.standard_normal(3 * N)).astype(np.float32)

    def make():
        lat = F.Lattice(nx, ny, nz, 0.57, storage="fp16s", model=model, smagorinsky=0.15,
                        mrt_rate=1.1, tasks=tasks)
        lat.upload_flags(flags)
        lat.upload_pops(pops)
        lat.upload_field("rho", rho)
        lat.upload_field("u", u)
        return lat

    for rounding in ("nearest", "stochastic"):
        a, b = pair(make, 9, -2, rounding)
        assert np.array_equal(a.download_pops(), b.download_pops())


@pytest.mark.parametrize("rounding", ["nearest", "stochastic"])
def test_tma_equals_direct_kernel_general_mrt(gpu_ok, rounding):
    """MRT whose non-shear rates differ runs the general moment form (the
    two-rate form needs one rate for all of them): the same bits in both
    kernels, from perturbed populations with bounce-back cells."""
    nx, ny, nz = 32, 24, 30
    N = nx * ny * nz
    rng = np.random.default_rng(11)
    flags = np.full(N, 2, dtype=np.uint8)
    flags[::7] = 4
    pops = (np.repeat(O.W, N) * (1 + 0.05 * rng.standard_normal(19 * N))).astype(np.float32)
    rates = [0, 1.1, 1.3, 0, 1.25, 0, 1.25, 0, 1.25, 1, 1.4, 1, 1.4, 1, 1, 1, 1.5, 1.5, 1.5]

    def make():
        lat = F.Lattice(nx, ny, nz, 0.55, storage="fp16s", model="mrt", mrt_rate=rates)
        lat.upload_flags(flags)
        lat.upload_pops(pops)
        return lat

    a, b = pair(make, 20, -2, rounding)
    assert np.array_equal(a.download_pops(), b.download_pops())


def test_tma_graph_and_autotune(gpu_ok):
    """CUDA-graph replay of the bulk-copy kernel equals plain launches; the
    autotuner times it among the candidates."""
    a = F.cavity(62, storage="fp16s")
    b = F.cavity(62, storage="fp16s")
    a.set_launch(4, -3, 4)
    b.set_launch(4, -3, 4)
    a.step(8, graph=True)
    b.step(8)
    assert np.array_equal(a.download_pops(), b.download_pops())
    c = F.cavity(62, storage="fp16s")
    (ty, ctas, v), ms, taken = c.autotune(trial_steps=1)
    assert ms > 0 and taken > 0
    c.device_status()


def test_tma_launch_rules(gpu_ok):
    with pytest.raises(F.FlbError):   # FP32 storage: not built
        F.cavity(30).set_launch(4, -2, 4)
    with pytest.raises(F.FlbError):   # rows not 16-byte aligned (pitch 52 halves)
        F.cavity(48, storage="fp16s").set_launch(4, -2, 4)
    with pytest.raises(F.FlbError):   # 2 cells per thread
        F.cavity(30, storage="fp16s").set_launch(4, -2, 2)
    with pytest.raises(F.FlbError):
        F.cavity(30, storage="fp16s").set_wait_limit(-1.0)


def test_tma_wait_that_gives_up_is_reported_and_the_handle_recovers(gpu_ok):
    """A tile whose stage is never signalled (the test hook withholds it): its
    consumers' waits run out after the 50 ms limit, the producer's wait for
    that stage too, the kernel ends early (the step is incomplete) and the
    status reads FLB_ERR_TIMEOUT once.  With the hook off and the state
    re-uploaded, the handle steps exactly like the direct kernel."""
    ni, steps = 62, 6
    ref = F.cavity(ni, tau=0.55, storage="fp16s")
    ref.set_launch(1, 0, 4)
    ref.step(steps)
    lat = F.cavity(ni, tau=0.55, storage="fp16s")
    start = lat.download_pops(np.float64)
    lat.set_launch(4, -2, 4)
    lat.set_wait_limit(0.05)
    lat.device_status()
    F._capi.call("flb_test_withhold_tile", lat._h, 150)   # a staged tile of CTA 2
    lat.step(1)
    with pytest.raises(F.FlbError) as e:
        lat.device_status()
    assert e.value.code == -4          # FLB_ERR_TIMEOUT
    lat.device_status()                # cleared
    F._capi.call("flb_test_withhold_tile", lat._h, -1)
    lat.set_wait_limit(2.0)
    lat.upload_pops(start)
    lat.step(steps)
    lat.device_status()
    assert np.array_equal(lat.download_pops(), ref.download_pops())


def test_results_of_a_default_handle_report_a_wait_that_gave_up(gpu_ok):
    """A caller who chose no launch shape runs the bulk-copy kernel at 128^3: until
    the status is read, every call that brings results to the host reports the
    incomplete step, and uploads, the way back, do not."""
    lat = F.cavity(126, tau=0.55, storage="fp16s")
    assert lat.get_launch() == (4, -2, 4)
    start = lat.download_pops(np.float64)
    lat.set_wait_limit(0.05)
    F._capi.call("flb_test_withhold_tile", lat._h, 150)
    lat.step(1)
    F._capi.call("flb_test_withhold_tile", lat._h, -1)
    lat.compute_rhou(2)
    for call in (lat.download_pops, lambda: lat.download_field("rho"),
                 lambda: lat.download_field("u"), lambda: lat.conservation(2),
                 lambda: lat.tolerance_u(2), lat.nonfinite, lambda: lat.autotune(1),
                 lambda: lat.vtk_body("rho")):
        with pytest.raises(F.FlbError) as e:
            call()
        assert e.value.code == -4      # FLB_ERR_TIMEOUT
    assert lat.get_launch() == (4, -2, 4)
    lat.upload_pops(start)
    with pytest.raises(F.FlbError):
        lat.device_status()
    lat.set_wait_limit(2.0)
    assert np.array_equal(lat.download_pops(np.float64), start)
    assert lat.conservation(2)[0] > 0


@pytest.mark.parametrize("ni,model,want", [
    (99, "bgk", (4, 0, 2)), (100, "bgk", (4, 0, 4)),    # 101^3, 102^3
    (104, "les", (4, 0, 2)),    # 106^3: the last size below the line
    (106, "bgk", (4, 0, 4)),    # 108^3: above it, rows not on 16-byte boundaries
    (106, "mrt", (4, 0, 2)),
    (108, "bgk", (4, 0, 4)),    # 110^3: rows of 112 with two cells of padding
    (108, "mrt", (4, 0, 4)),
    (110, "les", (4, -2, 4)),   # 112^3: none
    (110, "mrt", (4, -2, 4)),
    (118, "bgk", (4, 0, 4)),    # 120^3: the row ends at the same warps of every tile
    (126, "bgk", (4, -2, 4)),   # 128^3: the same, but in whole warps
    (158, "mrt", (4, -2, 4)),   # 160^3: in half warps
    (125, "les", (4, 0, 4)),    # 127^3: with padding
    (133, "bgk", (4, -2, 4)), (133, "les", (4, 0, 4)), (133, "mrt", (4, -2, 4)),  # 135^3
    (140, "bgk", (4, 0, 4)), (140, "mrt", (4, -2, 4)),                            # 142^3
    (131, "les", (4, 0, 4)), (131, "mrt", (4, -2, 4)),                            # 133^3
    (194, "mrt", (4, 0, 2)), (200, "mrt", (4, 0, 4)),   # 196^3, 202^3
    (204, "les", (4, -2, 4)),                           # 206^3
])
def test_default_shape_gives_the_direct_kernels_bits(gpu_ok, ni, model, want):
    """The shape the library picks by itself, on both sides of each line of its
    rule."""
    a, b = (F.cavity(ni, tau=0.55, storage="fp16s", model=model) for _ in range(2))
    assert a.get_launch() == want
    b.set_launch(1, 0, 4)
    a.step(6)
    b.step(6)
    a.device_status()
    assert np.array_equal(a.download_pops(), b.download_pops())


def set_model(lat, model):
    keys = (ctypes.c_uint8 * 3)(2, 4, 8)
    ops = (ctypes.c_uint8 * 3)(F._capi.OP_BULK, F._capi.OP_BOUNCEBACK, F._capi.OP_MOVINGWALL)
    F._capi.call("flb_set_tasks", lat._h, 3, keys, ops, model)


def test_default_shape_follows_the_model_of_a_live_handle(gpu_ok):
    """108^3 stored cells, whose rows do not suit the bulk copies: MRT takes 2 cells a
    thread there and BGK 4.  A handle that changes its model gives the bits of one
    whose shape is chosen; a tuning run that fails chooses nothing."""
    a, b = (F.cavity(106, tau=0.55, storage="fp16s", model="mrt") for _ in range(2))
    b.set_launch(1, 0, 4)
    for model, want in ((F._capi.MODEL_BGK, (4, 0, 4)), (F._capi.MODEL_MRT, (4, 0, 2)),
                        (F._capi.MODEL_BGK, (4, 0, 4))):
        set_model(a, model)
        set_model(b, model)
        assert a.get_launch() == want and b.get_launch() == (1, 0, 4)
        a.step(4)
        b.step(4)
        assert np.array_equal(a.download_pops(), b.download_pops())


def test_failed_autotune_leaves_the_default_in_charge(gpu_ok):
    lat = F.cavity(126, tau=0.55, storage="fp16s", model="mrt")
    lat.set_wait_limit(0.05)
    F._capi.call("flb_test_withhold_tile", lat._h, 150)
    lat.step(1)
    F._capi.call("flb_test_withhold_tile", lat._h, -1)
    with pytest.raises(F.FlbError) as e:
        lat.autotune(1)
    assert e.value.code == -4 and "gave up" in str(e.value)
    lat.set_wait_limit(2.0)
    assert lat.get_launch() == (4, -2, 4)
    F._capi.call("flb_test_wide_offsets", lat._h, 1)    # the default shape is picked again
    assert lat.get_launch() == (4, 0, 2)
