"""The neighbour walk where it can go wrong: the particle counts at which it takes another number of
particles per warp, partial warps, and runs whose candidates do not fit a warp's pool (they go
through it in segments).  Whole numbers and, with exact math, every record equal the oracle's bit
for bit."""
import numpy as np
import pytest

import akuaengine_gb300 as ak
from akuaengine_gb300 import LambdaCorrParams, PBFConfig, PBFSolver, scene
from test_gpu_parity import assert_grid_equal, assert_records_bitexact, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(cuda_lib):
    return cuda_lib


def first_of_block(n, seed):
    """The first n particles of a lattice block (a ragged last layer) in a box around it."""
    side = max(2, int(np.ceil(n ** (1.0 / 3.0))))
    sc = scene.dam_break((side, side, side), (2.0, 1.5, 1.5), seed=seed, jitter_frac=0.1)
    sc.particles = sc.particles[:n].copy()
    return sc


@pytest.mark.parametrize("where", [9, 31, 33, 65, "0.5-", "0.5+", "4-", "4+", "8-", "8+", "16-", "16+", "24-",
                                   "24+"])
def test_particles_per_warp_edges(where):
    """Counts around a warp and around the lines where the walk goes from 1 to 2 particles per warp
    and reaches 8 (1 x 12 and 8 x 12 per multiprocessor), then 16, 24 and 32 (8 x 24, 16 x 24 and
    24 x 24 in exact math)."""
    if isinstance(where, str):
        import torch

        sms = torch.cuda.get_device_properties(0).multi_processor_count
        n = int(float(where[:-1]) * 24 * sms) + (1 if where.endswith("+") else 0)
    else:
        n = where
    sc = first_of_block(n, seed=n)
    cfg, corr = PBFConfig(), LambdaCorrParams()
    g, ge = run_gpu(sc, cfg, corr, 1, ak.OPT_EXACT_MATH)
    o, oe = run_oracle(sc, cfg, corr, 1)
    assert_grid_equal(ge, oe, cfg.maxNeighbours)
    assert_records_bitexact(g, o)


@pytest.mark.parametrize("per_warp,warps_per_sm", [(8, 20), (12, 22), (20, 26), (28, 28)])
def test_particles_per_warp_edges_fast(per_warp, warps_per_sm):
    """One past the lines of fast math, where a warp takes 12, 16, 24 and 32 particles: the lists
    are those of the oracle (the first walk's positions do not depend on the math)."""
    import torch

    n = per_warp * warps_per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 1
    sc = first_of_block(n, seed=n)
    cfg, corr = PBFConfig(), LambdaCorrParams()
    _, ge = run_gpu(sc, cfg, corr, 1, 0)
    _, oe = run_oracle(sc, cfg, corr, 1)
    assert_grid_equal(ge, oe, cfg.maxNeighbours)


@pytest.mark.parametrize("shape", [(64, 16), (64, 32), (128, 48)])
@pytest.mark.parametrize("kind", ["wide_cell", "cluster", "small_table"])
def test_runs_longer_than_the_pool(shape, kind):
    """A walk cell of 2.5 h (sequences of thousands of candidates from buckets that are not the
    walk's cells), a cluster of 900 particles in a few cells (segments that end inside buckets,
    lists past the capacity), and the cluster under a table so small that its buckets are mixed
    and met twice."""
    sc = first_of_block(3000, seed=5)
    cfg, corr = PBFConfig(), LambdaCorrParams()
    if kind == "wide_cell":
        cfg.spatialHashCellSize = 0.25
    else:
        rng = np.random.default_rng(8)
        sc.particles["position"][:900] = (0.45 + rng.uniform(0.0, 0.17, (900, 3))).astype(np.float32)
    table = 512 if kind == "small_table" else None
    o, oe = run_oracle(sc, cfg, corr, 1, table_size=table)
    p = sc.particles.copy()
    with PBFSolver(sc.n, cfg, corr, options=ak.OPT_EXACT_MATH, table_size=table) as s:
        s.set_search_shape(*shape)
        s.step_host(p, sc.dt, sc.box_min, sc.box_max)
        ge = {"order": s.read_debug(ak.DEBUG_ORDER), "cnt": s.read_debug(ak.DEBUG_NEIGHBOUR_COUNTS),
              "nbr": s.read_debug(ak.DEBUG_NEIGHBOURS)}
    assert_grid_equal(ge, oe, cfg.maxNeighbours)
    assert_records_bitexact(p, o)


@pytest.mark.parametrize("exact", [True, False], ids=["exact", "fast"])
@pytest.mark.parametrize("where", ["8-", "8+", "4-", "4+", "2-", "2+"])
def test_lanes_per_particle_edges(where, exact):
    """Both sides of the lines where the pair kernels go from 8 to 4, 2 and 1 lanes per particle,
    with two masses.  Exact math: the oracle's records; fast math: those of the same particles
    stepped in a scene beyond every line (a far-away block makes up the number), whose kernels
    use one lane."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = {"8": (22 if exact else 10) * 32 * sms // 8, "4": (24 if exact else 18) * 32 * sms // 4,
           "2": (24 if exact else 18) * 32 * sms // 2}[where[0]]
    n = per + (1 if where.endswith("+") else 0)
    sc = first_of_block(n, seed=7)
    sc.particles["mass"][::3] = 0.8
    cfg, corr = PBFConfig(), LambdaCorrParams()
    if exact:
        g, ge = run_gpu(sc, cfg, corr, 1, ak.OPT_EXACT_MATH)
        o, oe = run_oracle(sc, cfg, corr, 1)
        assert_grid_equal(ge, oe, cfg.maxNeighbours)
        assert_records_bitexact(g, o)
        return
    # one table size, so the shared particles hash alike; the filler is out of everyone's reach
    table, extra = 1 << 24, 24 * 32 * sms
    fill = first_of_block(extra, seed=8).particles
    fill["position"][:, 0] += sc.box_max[0] + 5.0
    box_max = (sc.box_max[0] + 40.0,) + tuple(sc.box_max[1:])
    sc.particles["color"][:, 0] = np.arange(n) / np.float32(n)  # tell particles apart
    out = []
    for p in (sc.particles, np.concatenate([sc.particles, fill])):
        wide = scene.Scene(p.copy(), sc.box_min, box_max, sc.dt, "lanes")
        g, _ = run_gpu(wide, cfg, corr, 1, 0, table_size=table)
        own = g[g["position"][:, 0] < sc.box_max[0] + 2.0]
        out.append(own[np.lexsort((own["color"][:, 0],))])
    assert len(out[0]) == n == len(out[1])
    assert_records_bitexact(out[1], out[0])


@pytest.mark.parametrize("table_size", [None, 64], ids=["cells", "shared_buckets"])
def test_sparse_runs(table_size):
    """Spray: lone particles, pairs in one cell and in neighbouring cells, and clusters whose sequences
    lie around the 64 candidates that are tested without a cull; buckets of one cell each, and a
    table so small that lone particles find others in their buckets."""
    rng = np.random.default_rng(3)
    sc = first_of_block(1300, seed=3)
    pos = sc.particles["position"]
    pos[:] = rng.uniform(0.3, 5.7, pos.shape)  # 27,000 cells
    pos[100:300] = pos[300:500] + rng.uniform(-0.08, 0.08, (200, 3)).astype(np.float32)
    at = 600
    for k, size in enumerate((31, 32, 33, 63, 64, 65, 66, 128, 129)):
        corner = 0.5 + 0.6 * k
        pos[at:at + size] = corner + rng.uniform(0.005, 0.095, (size, 3))
        at += size
    sc.box_min, sc.box_max = (0.0, 0.0, 0.0), (6.0, 6.0, 6.0)
    cfg, corr = PBFConfig(), LambdaCorrParams()
    o, oe = run_oracle(sc, cfg, corr, 1, table_size=table_size)
    g, ge = run_gpu(sc, cfg, corr, 1, ak.OPT_EXACT_MATH, table_size=table_size)
    assert_grid_equal(ge, oe, cfg.maxNeighbours)
    assert_records_bitexact(g, o)


def pairs_out_of_sight(cell):
    """Lone particles within each other's reach, at rest.  A walk over cells of another size than the
    smoothing radius looks up buckets that need not hold the particle itself, so a single candidate
    may be its neighbour."""
    if cell in (0.2, 0.25):
        pos = np.array({0.2: [(0.41, 0.42, 0.41), (0.39, 0.39, 0.39)],
                        0.25: [(0.31, 0.05, 0.05), (0.24, 0.05, 0.05)]}[cell])
    else:
        rng = np.random.default_rng(12)
        axis = np.arange(6) * 0.35 + 0.1
        at = np.stack(np.meshgrid(axis, axis, axis, indexing="ij"), -1).reshape(-1, 3)
        at = at + rng.uniform(-0.05, 0.05, at.shape)
        d = rng.normal(size=at.shape)
        d *= rng.uniform(0.05, 0.095, (len(at), 1)) / np.linalg.norm(d, axis=1, keepdims=True)
        pos = np.concatenate([at, at + d])
    p = scene.lattice_block((len(pos), 1, 1), 0.0, (0.0, 0.0, 0.0))
    p["position"] = pos.astype(np.float32)
    return scene.Scene(p, (-1.0, -1.0, -1.0), (3.0, 3.0, 3.0), 0.0083, "pairs")


@pytest.mark.parametrize("exact", [True, False], ids=["exact", "fast"])
@pytest.mark.parametrize("cell", [0.09, 0.11, 0.13, 0.2, 0.25])
def test_lone_particles_under_another_walk_cell(cell, exact):
    sc = pairs_out_of_sight(cell)
    cfg, corr = PBFConfig(spatialHashCellSize=cell, gravity=(0.0, 0.0, 0.0)), LambdaCorrParams()
    o, oe = run_oracle(sc, cfg, corr, 1, table_size=1 << 20)
    assert oe["cnt"].any()  # the lists the oracle finds
    g, ge = run_gpu(sc, cfg, corr, 1, ak.OPT_EXACT_MATH if exact else 0, table_size=1 << 20)
    assert_grid_equal(ge, oe, cfg.maxNeighbours)
    if exact:
        assert_records_bitexact(g, o)
