"""The kernels that read the populations (fields, conservation sums, convergence
check) against FP64 sums of the downloaded populations, on rows that end inside,
at and one short of a chunk, with flags that split chunks, on several blocks and
with a porosity."""
import numpy as np
import pytest

import freelb_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

C = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1],
              [1, 1, 0], [-1, -1, 0], [1, 0, 1], [-1, 0, -1], [0, 1, 1], [0, -1, -1], [1, -1, 0],
              [-1, 1, 0], [1, 0, -1], [-1, 0, 1], [0, 1, -1], [0, -1, 1]], dtype=np.float64)


def moments(pops, n):
    f = np.asarray(pops, dtype=np.float64).reshape(19, n)
    rho = f.sum(0)
    return rho, (C.T @ f) / rho


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64", "fp32s"])
@pytest.mark.parametrize("dims", [(3, 3, 3), (5, 7, 6), (38, 5, 9), (63, 9, 8), (241, 4, 5)])
def test_readers_match_fp64_sums(gpu_ok, storage, dims):
    """A field value is a sum of 19 populations of size <= 0.4 in the arithmetic
    type: at most 19 roundings of a partial sum <= 1.1, i.e. 19 x 1.1 x 2^-24 for
    rho and as much over rho >= 0.9 for u (FP64: the same at 2^-53).  The sums
    are FP64 additions of the same terms."""
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(n)
    flags = rng.choice(np.array([1, 2, 4], dtype=np.uint8), size=n, p=[.2, .6, .2])
    lat = F.Lattice(*dims, 0.6, storage=storage)
    lat.upload_flags(flags)
    w = np.repeat(O.W, n)
    eps = 2.0 ** -53 if storage == "fp64" else 2.0 ** -24
    tol = 25 * eps
    hit = flags == 2
    old = np.zeros((3, n))
    lat.upload_field("rho", np.full(n, 7.0))
    for _ in range(2):
        lat.upload_pops(w * (1 + 0.02 * rng.standard_normal(19 * n)))
        pops = lat.download_pops(np.float64)
        rho, u = moments(pops, n)
        got_rho, got_u = lat.rhou(key=2, dtype=np.float64)
        got_u = got_u.reshape(n, 3).T
        assert np.max(np.abs(got_rho[hit] - rho[hit]), initial=0.0) < tol
        assert np.max(np.abs(got_u[:, hit] - u[:, hit]), initial=0.0) < tol
        assert np.all(got_rho[~hit] == 7.0) and np.all(got_u[:, ~hit] == 0.0)
        for key in (2, 6):
            m = (flags & key) != 0
            want = np.concatenate([[rho[m].sum()], (rho * u)[:, m].sum(1)])
            # FP32S adds its shift rho0 w_i in FP32 to the download, in FP64 here
            slack = 0.0 if storage == "fp64" else 19 * 2.0 ** -25 * max(1, m.sum())
            assert np.all(np.abs(lat.conservation(key) - want) <=
                          1e-12 * max(1.0, want[0]) + (slack if storage != "fp32" else 0.0))
        change = lat.tolerance_u(key=2)
        assert abs(change - np.max(np.abs(u - old)[:, hit], initial=0.0)) < 2 * tol
        old = np.where(hit, u, old)
    lat.close()


@pytest.mark.parametrize("storage,model", [("fp32", "bgk"), ("fp16s", "bgk"), ("fp64", "bgk"),
                                           ("fp32s", "bgk"), ("fp32", "brinkman"),
                                           ("fp64", "brinkman"), ("fp32s", "brinkman")])
def test_readers_on_blocks_and_with_porosity(gpu_ok, storage, model):
    """Three blocks of other shapes: the sums and the change of u go over all of
    them, the fields over each.  With a porosity the field u is the forced moment
    m / (rho + alpha / 2), of a smaller quotient and so within the same bound; the
    change of u is that of m / rho."""
    shapes = [(5, 7, 6), (38, 5, 9), (3, 3, 4)]
    rng = np.random.default_rng(5)
    lat = F.Lattice.blocks([s + (0, 0, 0) for s in shapes], 0.6, mode="independent",
                           storage=storage, model=model)
    tol = 25 * (2.0 ** -53 if storage == "fp64" else 2.0 ** -24)
    sums, change, cells = np.zeros(4), 0.0, 0
    want = []
    for k, (nx, ny, nz) in enumerate(shapes):
        n = nx * ny * nz
        flags = rng.choice(np.array([1, 2, 4], dtype=np.uint8), size=n, p=[.2, .6, .2])
        lat.upload_flags(flags, block=k)
        alpha = np.zeros(n)
        if model == "brinkman":
            alpha = rng.uniform(0, 2, n).astype(np.float32).astype(np.float64)
            lat.upload_field("alpha", alpha, block=k)
        lat.upload_pops(np.repeat(O.W, n) * (1 + 0.02 * rng.standard_normal(19 * n)), block=k)
        rho, u = moments(lat.download_pops(np.float64, block=k), n)
        hit = flags == 2
        want.append((hit, rho, u * rho / (rho + alpha / 2)))
        sums += np.concatenate([[rho[hit].sum()], (rho * u)[:, hit].sum(1)])
        change = max(change, np.max(np.abs(u[:, hit])))
        cells += int(hit.sum())
    lat.compute_rhou(2)
    for k, (hit, rho, u) in enumerate(want):
        got_u = lat.download_field("u", np.float64, block=k).reshape(-1, 3).T
        got_rho = lat.download_field("rho", np.float64, block=k)
        assert np.max(np.abs(got_rho[hit] - rho[hit])) < tol
        assert np.max(np.abs(got_u[:, hit] - u[:, hit])) < tol
    # FP16S and FP32S: the shift is added in FP32 for the download, in FP64 here
    slack = 19 * 2.0 ** -25 * cells if storage in ("fp16s", "fp32s") else 0.0
    assert np.all(np.abs(lat.conservation(2) - sums) <= 1e-12 * sums[0] + slack)
    assert abs(lat.tolerance_u(2) - change) < tol
