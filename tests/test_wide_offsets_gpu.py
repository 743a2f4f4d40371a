"""A single block with more than 2^32 population elements steps through the tile
kernel with 64-bit offsets, whatever its launch shape: the same path on small
lattices (flb_test_wide_offsets) against the single-block kernel, bit for bit."""
import numpy as np
import pytest

import freelb_b200 as F

pytestmark = pytest.mark.gpu


def lattices(storage, model, ni=34):
    a, b = (F.cavity(ni, tau=0.55, storage=storage, model=model) for _ in range(2))
    F._capi.call("flb_test_wide_offsets", b._h, 1)
    return a, b


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64", "fp32s"])
@pytest.mark.parametrize("model", ["bgk", "mrt", "les"])
def test_default_shape_steps(gpu_ok, storage, model):
    a, b = lattices(storage, model)
    for steps, graph in ((3, False), (4, True), (1, False)):
        a.step(steps, graph=graph)
        b.step(steps, graph=graph)
    assert np.array_equal(a.download_pops(), b.download_pops())


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64"])
def test_every_change_of_shape_gets_its_table(gpu_ok, storage):
    a, b = lattices(storage, "bgk")
    v = 2
    for shape in ((1, 0, v), (8, 0, v), (2, 4, v), (2, 0, v if storage == "fp64" else 4)):
        b.set_launch(*shape)
        a.step(3)
        b.step(3)
        assert np.array_equal(a.download_pops(), b.download_pops())
    taken = b.autotune(trial_steps=1)[2]
    a.step(taken)
    b.step(3)
    a.step(3)
    assert np.array_equal(a.download_pops(), b.download_pops())


def test_staged_kernels_are_refused(gpu_ok):
    lat = F.cavity(30, storage="fp16s")
    F._capi.call("flb_test_wide_offsets", lat._h, 1)
    for ctas in (-1, -2, -3):
        with pytest.raises(F.FlbError):
            lat.set_launch(4, ctas, 4)


def test_adjoint_recompute(gpu_ok):
    """The backward sweep's recomputed steps take the same path as the forward's."""
    out = []
    for lat in lattices("fp32s", "brinkman", ni=20):
        lat.upload_field("alpha", np.full(lat.N, 0.05))
        J = lat.adjoint_forward(12, 4)
        out.append((J,) + lat.adjoint_backward())
    (ja, ga, ta, ua), (jb, gb, tb, ub) = out
    assert ja == jb and np.array_equal(ga, gb) and (ta, ua) == (tb, ub)
