"""GPU tests of multi-block lattices: device halo exchange (uneven blocks of
one cavity), the batched ensemble of independent cavities, launch-shape
control, the autotuner and CUDA-graph stepping."""
import numpy as np
import pytest

import freelb_b200 as F
from conftest import golden, rel_maxnorm
from freelb_b200 import geometry as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def gpu_blocks(ni, blocks, storage="fp32", tau=0.53, ulid=0.1, model="bgk"):
    n = ni + 2
    flags = F.cavity_flags(ni)
    lat = F.Lattice.blocks(G.block_tuples(blocks), tau, mode="halo", storage=storage,
                           model=model)
    real = lat.real
    u = np.zeros((n ** 3, 3), dtype=real)
    u[flags == 8, 0] = real(ulid)
    for k, b in enumerate(blocks):
        lat.upload_flags(G.slice_block(flags, n, b), block=k)
        lat.upload_field("u", G.slice_block(u, n, b, comps=3), block=k)
    return lat


@pytest.mark.parametrize("name", ["blocks_bgk_f64_n12_s30", "blocks_bgk_f32_n12_s30"])
def test_blocks_match_reference_multiblock_golden(gpu_ok, name):
    g = golden(name)
    ni, _, _, steps, seed = g["params"]
    blocks = G.uneven_blocks(int(ni), edges=tuple(int(e) for e in g["edges"]), seed=int(seed))
    storage = "fp64" if "f64" in name else "fp32"
    lat = gpu_blocks(int(ni), blocks, storage)
    assert lat.halo_count() > 0
    lat.step(int(steps))
    lat.compute_rhou(2)
    tol = 1e-12 if storage == "fp64" else 1e-5
    pops = np.concatenate([lat.download_pops(block=k) for k in range(len(blocks))])
    ref = np.concatenate([g[f"pops_b{k}"] for k in range(len(blocks))])
    assert rel_maxnorm(pops, ref) < tol
    u = np.concatenate([lat.download_field("u", block=k) for k in range(len(blocks))])
    uref = np.concatenate([g[f"u_b{k}"] for k in range(len(blocks))])
    assert rel_maxnorm(u, uref) < tol
    for k in range(len(blocks)):
        assert np.array_equal(lat.download_flags(block=k), g[f"flags_b{k}"])


@pytest.mark.parametrize("model", ["bgk", "mrt", "les"])
@pytest.mark.parametrize("tile_y,ctas,vec", [(8, 0, 4), (2, 8, 2), (1, 0, 2), (4, 16, 4)])
def test_blocks_vs_single_block_bitwise_on_fluid(gpu_ok, tile_y, ctas, vec, model):
    """Uneven blocks with device halos reproduce the single-block run exactly on
    fluid cells, for every launch shape and model (MRT in its two-rate form)."""
    ni = 40
    blocks = G.uneven_blocks(ni, edges=(8, 12, 16), seed=5)
    lat = gpu_blocks(ni, blocks, "fp32", model=model)
    lat.set_launch(tile_y, ctas, vec)
    lat.step(40)
    one = F.cavity(ni, model=model)
    one.step(40)
    n = ni + 2
    P = one.download_pops().reshape(19, n, n, n)
    for k, b in enumerate(blocks):
        pb = lat.download_pops(block=k).reshape(19, b["nz"], b["ny"], b["nx"])
        fb = G.slice_block(F.cavity_flags(ni), n, b).reshape(b["nz"], b["ny"], b["nx"])
        ps = P[:, b["oz"]:b["oz"] + b["nz"], b["oy"]:b["oy"] + b["ny"], b["ox"]:b["ox"] + b["nx"]]
        assert np.array_equal(pb[:, fb == 2], ps[:, fb == 2])


@pytest.mark.parametrize("model", ["bgk", "mrt", "les"])
@pytest.mark.parametrize("tile_y,ctas,vec", [(8, 0, 4), (2, 8, 2), (4, 16, 4)])
def test_fp16s_blocks_vs_single_block_bitwise_on_fluid(gpu_ok, model, tile_y, ctas, vec):
    """FP16S storage: the multi-block tile kernel (32-bit offsets) and the
    single-block kernel give the same bits on fluid cells."""
    ni = 40
    blocks = G.uneven_blocks(ni, edges=(8, 12, 16), seed=7)
    lat = gpu_blocks(ni, blocks, "fp16s", tau=0.55, model=model)
    lat.set_launch(tile_y, ctas, vec)
    lat.step(30)
    one = F.cavity(ni, tau=0.55, storage="fp16s", model=model)
    one.step(30)
    n = ni + 2
    P = one.download_pops().reshape(19, n, n, n)
    for k, b in enumerate(blocks):
        pb = lat.download_pops(block=k).reshape(19, b["nz"], b["ny"], b["nx"])
        fb = G.slice_block(F.cavity_flags(ni), n, b).reshape(b["nz"], b["ny"], b["nx"])
        ps = P[:, b["oz"]:b["oz"] + b["nz"], b["oy"]:b["oy"] + b["ny"], b["ox"]:b["ox"] + b["nx"]]
        assert np.array_equal(pb[:, fb == 2], ps[:, fb == 2]), (model, k)


def test_blocks_vs_oracle_multiblock_fp64(gpu_ok):
    ni = 18
    blocks = G.uneven_blocks(ni, edges=(4, 6, 8), seed=9)
    lat = gpu_blocks(ni, blocks, "fp64", tau=0.56, ulid=0.08)
    mb = O.MultiBlock(blocks, O.cavity_flags(ni), ni + 2, tau=0.56, ulid=0.08, dtype=np.float64)
    lat.step(33)
    mb.step(33)
    ours = np.concatenate([lat.download_pops(block=k) for k in range(len(blocks))])
    ref = np.concatenate([m.pops for m in mb.lats])
    assert rel_maxnorm(ours, ref) < 1e-12


def ensemble(sizes, taus, storage="fp32", ulid=0.1):
    lat = F.Lattice.blocks([(n + 2, n + 2, n + 2, 0, 0, 0, 1.0 / t) for n, t in zip(sizes, taus)],
                           0.6, mode="independent", storage=storage)
    for k, n in enumerate(sizes):
        fl = F.cavity_flags(n)
        u = np.zeros(((n + 2) ** 3, 3), dtype=lat.real)
        u[fl == 8, 0] = lat.real(ulid)
        lat.upload_flags(fl, block=k)
        lat.upload_field("u", u, block=k)
    return lat


@pytest.mark.parametrize("graph", [False, True])
def test_ensemble_each_cavity_matches_single(gpu_ok, graph):
    """Batched independent cavities, each with its own tau, match one-at-a-time runs."""
    rng = np.random.default_rng(1)
    sizes = [int(v) for v in rng.integers(6, 20, size=9)]
    taus = [0.5 + 3 * 0.1 * n / float(np.exp(rng.uniform(np.log(100), np.log(3000))))
            for n in sizes]
    lat = ensemble(sizes, taus)
    lat.step(25, graph=graph)
    for k, (n, t) in enumerate(zip(sizes, taus)):
        ref = O.cavity(n, tau=t, ulid=0.1)
        ref.step(25)
        assert rel_maxnorm(lat.download_pops(block=k), ref.pops) < 1e-5, (k, n, t)


@pytest.mark.parametrize("graph", [False, True])
def test_fp16s_ensemble_each_cavity_equals_single(gpu_ok, graph):
    """FP16S storage: the batched cavities, each with its own tau, give the bits
    of one FP16S handle per cavity (the 32-bit tile kernel against the
    single-block kernel)."""
    rng = np.random.default_rng(2)
    sizes = [int(v) for v in rng.integers(6, 24, size=7)]
    taus = [0.5 + 3 * 0.1 * n / float(np.exp(rng.uniform(np.log(100), np.log(3000))))
            for n in sizes]
    lat = ensemble(sizes, taus, storage="fp16s")
    lat.step(25, graph=graph)
    for k, (n, t) in enumerate(zip(sizes, taus)):
        one = F.cavity(n, tau=t, ulid=0.1, storage="fp16s")
        one.step(25)
        assert np.array_equal(lat.download_pops(block=k), one.download_pops()), (k, n, t)
        one.close()


def test_graph_step_equals_plain_step(gpu_ok):
    a = F.cavity(30)
    b = F.cavity(30)
    a.step(17)
    b.step(17, graph=True)
    assert np.array_equal(a.download_pops(), b.download_pops())
    a.step(4, graph=True)
    b.step(4)
    assert np.array_equal(a.download_pops(), b.download_pops())


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64"])
def test_autotune_keeps_results_exact(gpu_ok, storage):
    a = F.cavity(36, storage=storage)
    b = F.cavity(36, storage=storage)
    (ty, c, v), ms, taken = a.autotune(trial_steps=2)
    assert ty in (1, 2, 4, 8) and c in (-3, -2, -1, 0, 8, 16, 32) and ms > 0 and taken > 0
    assert c >= 0 or storage == "fp16s"
    assert v in ((1, 2) if storage == "fp64" else (2, 4))
    assert a.get_launch() == (ty, c, v)
    b.step(taken)
    a.step(5)
    b.step(5)
    assert np.array_equal(a.download_pops(), b.download_pops())


def test_set_launch_rejects_bad_shapes(gpu_ok):
    a = F.cavity(8)
    with pytest.raises(F.FlbError):
        a.set_launch(3, 0)
    with pytest.raises(F.FlbError):
        a.set_launch(8, -1)
    with pytest.raises(F.FlbError):
        a.set_launch(8, 0, 1)     # FP32 builds 2 or 4 cells per thread


@pytest.mark.parametrize("storage,vec", [("fp32", 2), ("fp32", 4), ("fp16s", 2), ("fp16s", 4),
                                         ("fp64", 1), ("fp64", 2)])
def test_every_vector_width_matches_oracle(gpu_ok, storage, vec):
    lat = F.cavity(21, tau=0.55, storage=storage)
    lat.set_launch(4, 0, vec)
    lat.step(30)
    ref = O.cavity(21, tau=0.55, dtype=np.float64 if storage == "fp64" else np.float32)
    ref.step(30)
    tol = {"fp32": 1e-5, "fp64": 1e-12, "fp16s": 2e-3}[storage]
    assert rel_maxnorm(lat.download_pops(), ref.pops) < tol


@pytest.mark.parametrize("model", ["bgk", "mrt", "les"])
@pytest.mark.parametrize("storage,widths", [("fp32", (2, 4)), ("fp16s", (2, 4)), ("fp64", (1, 2)),
                                            ("fp32s", (2, 4))])
@pytest.mark.parametrize("ni", [21, 30])
def test_vector_widths_are_bitwise_equal(gpu_ok, storage, widths, ni, model):
    """Every cell's update is the same function of its 19 sources whatever the
    cells per thread or launch shape (direct, persistent tile kernel), so they
    agree bit for bit (ragged rows and row ends included): the autotuner's pick
    never changes a result."""
    out = []
    for v in widths:
        for shape in ((2, 0, v), (8, 16, v)):
            lat = F.cavity(ni, tau=0.55, storage=storage, model=model)
            lat.set_launch(*shape)
            lat.step(25)
            out.append(lat.download_pops())
    for o in out[1:]:
        assert np.array_equal(out[0], o)


@pytest.mark.parametrize("storage,tol", [("fp64", 1e-12), ("fp32", 1e-5), ("fp16s", 2e-3)])
def test_full_halo_matches_oracle(gpu_ok, storage, tol):
    """flb_set_halo_mode(FULL): all 19 populations of every overlap cell from its
    owner (NormalFullCommunicate / NormalAllCommunicate), against the oracle's
    restatement (itself pinned to the reference's run)."""
    ni, steps = 16, 20
    blocks = G.uneven_blocks(ni, edges=(4, 6, 8), seed=3)
    lat = gpu_blocks(ni, blocks, storage)
    normal = lat.halo_count()
    lat.set_halo_mode("full")
    assert lat.halo_count() > normal
    lat.step(steps)
    dt = np.float32 if storage == "fp32" else np.float64  # FP16S against FP64
    mb = O.MultiBlock(blocks, O.cavity_flags(ni), ni + 2, dtype=dt, full=True)
    mb.step(steps)
    pops = np.concatenate([lat.download_pops(block=k) for k in range(len(blocks))])
    want = np.concatenate([mb.lats[k].pops for k in range(len(blocks))])
    assert rel_maxnorm(pops, want) < tol
    lat.set_halo_mode("normal")
    assert lat.halo_count() == normal


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64", "fp32s"])
@pytest.mark.parametrize("dims", [(3, 3, 3), (5, 9, 4), (100, 60, 50), (100, 60, 51)])
def test_small_lattice_form_equals_the_tile_kernel(gpu_ok, storage, dims):
    """The step kernel's form for small lattices (up to 300,000 padded cells: the
    third shape is the last of them) against the tile kernel, bit for bit, on
    every row near the first and last planes and with every op."""
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(n)
    flags = rng.choice(np.array([1, 2, 4, 8, 16], dtype=np.uint8), size=n, p=[.1, .6, .1, .1, .1])
    tasks = ((2, "bulk"), (4, "bounceback"), (8, "movingwall"), (16, "field_bgk"))
    pops = np.repeat(O.W, n) * (1 + 0.05 * rng.standard_normal(19 * n))
    u = 0.03 * rng.standard_normal(3 * n)
    out = []
    for shape in ((4, 0, 2), (8, 16, 2)):
        lat = F.Lattice(*dims, 0.57, storage=storage, tasks=tasks)
        lat.upload_flags(flags)
        lat.upload_pops(pops)
        lat.upload_field("u", u)
        lat.set_launch(*shape)
        lat.step(5)
        out.append(lat.download_pops())
        lat.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("dims,want", [((100, 60, 50), (4, 0, 2)), ((100, 60, 51), (2, 0, 2)),
                                       ((150, 150, 200), (2, 0, 4)), ((160, 150, 190), (2, 0, 2))])
def test_default_fp32_shape_equals_the_tile_kernel(gpu_ok, dims, want):
    """The shapes the library picks for FP32 BGK, on both sides of each line of
    its rule, against the tile kernel."""
    out = []
    for chosen in (None, (8, 16, 2)):
        lat = F.Lattice(*dims, 0.55)
        flags = np.ones(dims[::-1], np.uint8)
        flags[1:-1, 1:-1, 1:-1] = 4
        flags[2:-2, 2:-2, 2:-2] = 2
        flags[-2, 2:-2, 2:-2] = 8
        lat.upload_flags(flags)
        u = np.zeros((flags.size, 3), np.float32)
        u[flags.reshape(-1) == 8, 0] = 0.1
        lat.upload_field("u", u)
        if chosen:
            lat.set_launch(*chosen)
        else:
            assert lat.get_launch() == want
        lat.step(4)
        out.append(lat.download_pops())
        lat.close()
    assert np.array_equal(out[0], out[1])


def test_autotune_leaves_the_winner_ready_to_be_captured(gpu_ok):
    """After a tuning run the block table is that of the shape it kept, so a
    caller's capture of the next steps allocates and copies nothing."""
    import torch
    a, b = (gpu_blocks(40, G.uneven_blocks(40, edges=(8, 12, 16), seed=2)) for _ in range(2))
    taken = a.autotune(trial_steps=1)[2]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        a.step(2, stream)
    graph.replay()
    torch.cuda.synchronize()
    b.step(taken + 2)
    for k in range(a.nblocks):
        assert np.array_equal(a.download_pops(block=k), b.download_pops(block=k))


GENERAL = [0, 1.1, 1.3, 0, 1.25, 0, 1.25, 0, 1.25, 1, 1.4, 1, 1.4, 1, 1, 1, 1.5, 1.5, 1.5]


@pytest.mark.parametrize("storage,kw,count,want", [
    ("fp32", {}, 1, (4, 0, 2)), ("fp32", {}, 2, (4, 32, 4)),
    ("fp32", {"model": "les"}, 2, (4, 32, 4)),
    ("fp32", {"model": "mrt"}, 1, (4, 0, 2)), ("fp32", {"model": "mrt"}, 2, (4, 32, 4)),
    ("fp32", {"model": "mrt", "mrt_rate": GENERAL}, 5, (4, 0, 2)),
    ("fp32", {"model": "mrt", "mrt_rate": GENERAL}, 6, (4, 32, 4)),
    ("fp16s", {}, 1, (4, 0, 2)), ("fp16s", {"model": "mrt"}, 2, (4, 32, 4)),
    ("fp16s", {"model": "mrt", "mrt_rate": GENERAL}, 2, (4, 32, 4)),
    ("fp64", {}, 1, (4, 0, 1)), ("fp64", {}, 2, (4, 32, 2)), ("fp32s", {"model": "mrt"}, 2, (4, 0, 2)),
])
def test_default_shapes_of_many_blocks(gpu_ok, storage, kw, count, want):
    """Cavities of 60^3 stored cells (216,000 each) on both sides of the rule's
    lines, against another shape, bit for bit."""
    flags = F.cavity_flags(58)
    u = np.zeros((flags.size, 3))
    u[flags == 8, 0] = 0.1
    out = []
    for chosen in (None, (8, 0, 2)):
        lat = F.Lattice.blocks([(60, 60, 60, 0, 0, 0)] * count, 0.55, mode="independent",
                               storage=storage, **kw)
        for k in range(count):
            lat.upload_flags(flags, block=k)
            lat.upload_field("u", u, block=k)
        if chosen:
            lat.set_launch(*chosen)
        else:
            assert lat.get_launch() == want
        lat.step(6)
        out.append([lat.download_pops(block=k) for k in range(count)])
        lat.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("storage,model,vecs", [
    ("fp32", "bgk", (2, 4)), ("fp32", "mrt", (2, 4)), ("fp32", "les", (2, 4)),
    ("fp32", "brinkman", (2, 4)), ("fp32s", "bgk", (2, 4)), ("fp32s", "mrt", (2, 4)),
    ("fp32s", "les", (2, 4)), ("fp32s", "brinkman", (2, 4)), ("fp64", "bgk", (1, 2)),
    ("fp64", "mrt", (1, 2)), ("fp64", "les", (1, 2)), ("fp64", "brinkman", (1, 2)),
])
def test_early_form_of_the_tile_kernel_gives_the_usual_ones_bits(gpu_ok, storage, model, vecs):
    """Plain steps of a small handle run the tile kernel's early form, captured ones
    (a graph's launches are ordered as usual) the other; FP64, which has the early
    form alone, against the single-block kernel.  Every op, on ragged blocks."""
    tasks = ((2, "bulk"), (4, "bounceback"), (8, "movingwall"), (16, "field_bgk"))
    shapes = [(37, 20, 18), (24, 30, 19), (9, 7, 50)]
    for v in vecs:
        for ctas in (0, 8):
            out = []
            for graph in (False, True):
                rng = np.random.default_rng(v)
                lat = F.Lattice.blocks([d + (0, 0, 0) for d in shapes], 0.57,
                                       mode="independent", storage=storage, model=model,
                                       tasks=tasks)
                ones = []
                for k, d in enumerate(shapes):
                    n = d[0] * d[1] * d[2]
                    flags = rng.choice(np.array([1, 2, 4, 8, 16], dtype=np.uint8), size=n,
                                       p=[.1, .6, .1, .1, .1])
                    pops = np.repeat(O.W, n) * (1 + 0.05 * rng.standard_normal(19 * n))
                    u, alpha = 0.03 * rng.standard_normal(3 * n), rng.uniform(0, 1, n)
                    one = F.Lattice(*d, 0.57, storage=storage, model=model, tasks=tasks)
                    for to, b in ((lat, k), (one, 0)):
                        to.upload_flags(flags, block=b)
                        to.upload_pops(pops, block=b)
                        to.upload_field("u", u, block=b)
                        if model == "brinkman":
                            to.upload_field("alpha", alpha, block=b)
                    ones.append(one)
                lat.set_launch(4, ctas, v)
                lat.step(6, graph=graph)
                out.append([lat.download_pops(block=k) for k in range(len(shapes))])
                if storage == "fp64":
                    for one in ones:
                        one.set_launch(4, 0, v)
                        one.step(6)
                    out.append([one.download_pops() for one in ones])
            for o in out[1:]:
                assert all(np.array_equal(a, b) for a, b in zip(out[0], o))
