"""The tile-based sampler and measurement (planes as 8×8 tiles of the upper triangle) at the
edges of their ranges: sides around multiples of 8, 32 and 64, one and several planes, few
and many samples, every exchange mix; and the square-plane sampler on the models left to it."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle_lib as ol
from mvmc_lib import lattice, mvmc

pytestmark = pytest.mark.gpu


def inputs(tmp_path, lx, ly, n_up, nmp=1, nsp=1, **kw):
    shifts = [(0, 0), (1, 0), (0, 1), (1, 1)] if ly > 1 else [(0, 0), (1, 0), (2, 0), (3, 0)]
    args = dict(n_up=n_up, nmp=nmp, nsp_gauss_leg=nsp, shifts=shifts, samples=2, warmup=2, interval=3)
    args.update(kw)
    return lattice().write_inputs(str(tmp_path), lx, ly, **args)[:2]


@pytest.mark.parametrize("lx,ly,n_up,nmp,nsp,kw", [
    (4, 1, 1, 1, 1, {}),                       # n = 2: one tile, six of its rows padding
    (9, 1, 4, 1, 1, {}),                       # n = 8: one full tile
    (12, 1, 5, 1, 1, dict(ex_path=0)),         # n = 10, hops only (eight proposals a batch)
    (8, 4, 16, 1, 1, dict(ex_path=2)),         # n = 32, exchanges only: the last side of 128 threads
    (6, 6, 17, 1, 1, {}),                      # n = 34: the first side of 512 threads
    (5, 5, 11, 2, 2, {}),                      # four planes: a refresh sweeps a plane per warp
    (8, 8, 32, 4, 2, dict(sub=(2, 1))),        # n = 64, eight planes
    (9, 8, 33, 1, 2, {}),                      # n = 66: above the warp sweep
    (14, 13, 84, 1, 1, dict(interval=1)),      # n = 168
])
def test_tile_sampler_reproduces_the_oracle_chains(tmp_path, lx, ly, n_up, nmp, nsp, kw):
    """Saved configurations, counters and draw counts of three chains equal the oracle's:
    batches of speculative proposals leave the chain as one proposal after the other."""
    nl, init = inputs(tmp_path, lx, ly, n_up, nmp, nsp, **kw)
    _, ref = ol.opt_step1_walkers(nl, 3, seed=11, initial_def=init)
    eng = mvmc().Engine(nl, initial_def=init, walkers=3, precision=64, seed=11)
    eng.sample()
    got = eng.samples()
    for key in ("ele_idx", "proj_cnt", "counter", "draws"):
        assert got[key].tolist() == ref[key].tolist(), key
    assert eng.status() == 0


@pytest.mark.parametrize("lx,ly,n_up,nmp,nsp,walkers", [
    (6, 6, 17, 1, 1, 160),     # n = 34: 256 threads, the block sweeps
    (8, 4, 16, 4, 1, 160),     # n = 32, four planes: 256 threads, a plane per warp
    (8, 8, 32, 4, 1, 160),     # n = 64
    (9, 8, 33, 1, 1, 160),     # n = 66
    (16, 8, 64, 1, 1, 160),    # n = 128: the last side of 256 threads
    (8, 4, 16, 4, 1, 460),     # n = 32: 128 threads, a column per lane
    (6, 6, 17, 1, 1, 460),     # n = 34: 128 threads, two columns per lane
    (8, 8, 32, 1, 2, 460),     # n = 64
])
def test_tile_sampler_with_several_walkers_per_sm(tmp_path, lx, ly, n_up, nmp, nsp, walkers):
    """More walkers than SMs take 256 or 128 threads each. A chain depends on its seed alone:
    the first three equal the oracle's."""
    nl, init = inputs(tmp_path, lx, ly, n_up, nmp, nsp)
    _, ref = ol.opt_step1_walkers(nl, 3, seed=11, initial_def=init)
    eng = mvmc().Engine(nl, initial_def=init, walkers=walkers, precision=64, seed=11)
    eng.sample()
    got = eng.samples()
    for key in ("ele_idx", "proj_cnt", "counter", "draws"):
        assert got[key].reshape(walkers, -1)[:3].ravel().tolist() == ref[key].tolist(), key
    assert eng.status() == 0


SQUARE_PLANES = [
    (16, 1, 8, 16, 4, "auto"),    # n = 16, 64 planes: squares in shared memory, 128 threads
    (6, 6, 17, 18, 1, "auto"),    # n = 34, 18 planes: squares, 512 threads
    (8, 8, 32, 16, 1, "auto"),    # n = 64, 16 planes: planes in L2
    (16, 16, 113, 1, 1, "auto"),  # n = 226: the first side without tiles
    (16, 16, 128, 1, 1, "auto"),  # n = 256: the half-filled lattice
    (8, 8, 32, 4, 2, "global"),   # planes in L2 on request
    (11, 10, 54, 1, 1, "global"),
]


def square_plane_chains(path, lx, ly, n_up, nmp, nsp):
    shifts = [(x, y) for y in range(ly) for x in range(lx)]
    nl, init, _ = lattice().write_inputs(path, lx, ly, n_up=n_up, nmp=nmp, nsp_gauss_leg=nsp, shifts=shifts, samples=2,
                                         warmup=2, interval=2)
    _, ref = ol.opt_step1_walkers(nl, 3, seed=11, initial_def=init)
    eng = mvmc().Engine(nl, initial_def=init, walkers=3, precision=64, seed=11)
    eng.sample()
    got = eng.samples()
    for key in ("ele_idx", "proj_cnt", "counter", "draws"):
        assert got[key].tolist() == ref[key].tolist(), key
    e = eng.measure()[0]
    assert np.allclose(e, ref["energy"], rtol=1e-9)
    assert eng.status() == 0


@pytest.mark.parametrize("lx,ly,n_up,nmp,nsp,residency", SQUARE_PLANES)
def test_square_plane_sampler_reproduces_the_oracle_chains(tmp_path, lx, ly, n_up, nmp, nsp, residency):
    """FP64 models whose planes do not fit as tiles, or are asked to stay in L2, run on square
    planes. In a process of its own: the residency is read once."""
    code = ("import test_tile_kernels_gpu as t; "
            f"t.square_plane_chains({str(tmp_path)!r}, {lx}, {ly}, {n_up}, {nmp}, {nsp})")
    env = dict(os.environ, MVMC_B200_RESIDENCY=residency)
    run = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.abspath(__file__)), env=env,
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]


@pytest.mark.parametrize("lx,ly,n_up,nmp,nsp,walkers", [
    (8, 8, 32, 4, 2, 700),     # n = 64, eight planes: two warps per sample
    (8, 8, 32, 4, 2, 40),      # the same, eight warps per sample
    (8, 8, 31, 4, 2, 700),     # n = 62
    (7, 5, 17, 4, 2, 40),      # n = 34
    (8, 4, 16, 4, 2, 700),     # n = 32
    (8, 4, 4, 4, 2, 700),      # n = 8: one tile
    (9, 8, 33, 1, 2, 9),       # n = 66, 256 threads
    (11, 12, 64, 1, 1, 9),     # n = 128
    (11, 12, 65, 1, 1, 9),     # n = 130, 512 threads
    (16, 14, 111, 1, 1, 9),    # n = 222
])
def test_tile_measurement_matches_the_square_planes(tmp_path, monkeypatch, lx, ly, n_up, nmp, nsp, walkers):
    """O rows, energies and ln|Psi| of the same samples from tiles and from the in-place sweep
    of square planes. Two sweeps of one plane differ by its condition number (below 1e5 here)
    times the rounding of n/2 steps, 1e5 · 128 · 1e-16 ≈ 1e-9 relative."""
    nl, init = inputs(tmp_path, lx, ly, n_up, nmp, nsp, interval=1, samples=1)
    eng = mvmc().Engine(nl, initial_def=init, walkers=walkers, precision=64, seed=5)
    eng.sample()
    rows = {}
    for mode in ("tiles", "l2"):
        monkeypatch.setenv("MVMC_B200_MEASURE", mode)
        e, ho, oo = eng.measure()
        rows[mode] = (eng.o_store(), eng.local_energies(), eng.log_amplitudes(), e, ho, oo)
    assert eng.status() == 0
    for a, b in zip(rows["tiles"], rows["l2"]):
        assert np.max(np.abs(a - b)) <= 1e-9 * max(1.0, np.max(np.abs(b)))


@pytest.mark.parametrize("sites,walkers", [
    (2, 64),     # n = 4, a warp per plane, a column per lane
    (18, 450),   # n = 36, two columns per lane
    (34, 64),    # n = 68, eight warps per panel
    (34, 160),   # four warps per panel
])
def test_pivot_is_the_largest_entry(tmp_path, monkeypatch, sites, walkers):
    """Planes of 2×2 blocks ((x, v), (b, 0)), v = x + 2⁻²⁰, in each walker's own electron order. The
    inverse has a zero where x stands, which the sweep keeps exactly with v as pivot; with x,
    where it comes first, it becomes the rounding of 1/x − v·(1/x)·(1/v). Sites are full and
    only exchanges are tried, so no move is made and the resident measurement shows the
    sampler's sweep."""
    nl, init = inputs(tmp_path, sites, 1, sites, sub=(sites, 1), ex_path=2, interval=1, samples=1, warmup=1)
    for mode, resident in (("l2", 0), ("tiles", 0), ("tiles", 1)):
        monkeypatch.setenv("MVMC_B200_MEASURE", mode)
        eng = mvmc().Engine(nl, initial_def=init, walkers=walkers, precision=64, seed=5, measure_resident=resident)
        p = np.zeros(eng.dims["npara"])
        f = p[eng.dims["nproj"]:].reshape(sites, sites)  # [site, displacement]
        f[0::2, 0], f[0::2, 1], f[1::2, sites - 1] = 0.9, 0.9 + 2.0 ** -20, 0.6
        eng.set_parameters(p)
        eng.sample()
        eng.measure()
        assert eng.status() == 0
        o = eng.o_store()[:, 1 + eng.dims["nproj"]:].reshape(walkers, sites, sites)
        assert np.all(o[:, 0::2, 1] != 0.0) and np.all(o[:, 0::2, 0] == 0.0), (mode, resident)


@pytest.mark.parametrize("lx,ly,n_up,nmp,nsp,walkers", [
    (8, 8, 32, 4, 1, 700),     # n = 64, four planes: the digits of the square planes
    (8, 4, 16, 16, 2, 40),     # n = 32, 32 planes, few samples: the squares are faster
])
def test_measurement_on_square_planes_beside_the_tiles(tmp_path, monkeypatch, lx, ly, n_up, nmp, nsp, walkers):
    """Where the choice falls on the square planes the results are theirs bit for bit."""
    shifts = [(x, y) for y in range(ly) for x in range(lx)]
    nl, init = inputs(tmp_path, lx, ly, n_up, nmp, nsp, shifts=shifts, interval=1, samples=1)
    eng = mvmc().Engine(nl, initial_def=init, walkers=walkers, precision=64, seed=5)
    eng.sample()
    rows = []
    for mode in ("tiles", "l2"):
        monkeypatch.setenv("MVMC_B200_MEASURE", mode)
        eng.measure()
        rows.append(eng.o_store())
    assert np.array_equal(*rows)


def hoppings_within(path, ns, reach):
    """Rewrite trans.def: every site hops to its `reach` next sites on either side (in the
    order of the site index), both spins."""
    lines = []
    for i in range(ns):
        for d in range(1, reach + 1):
            for j in ((i + d) % ns, (i - d) % ns):
                lines += [f"{i:5d} {s:5d} {j:5d} {s:5d} {0.1 / d: .15f} {0.0: .15f}\n" for s in (0, 1)]
    lattice()._def_file(str(path / "trans.def"), "NTransfer", len(lines), "".join(lines))


@pytest.mark.parametrize("lx,ly,n_up,nmp,nsp,reach,walkers", [
    (8, 8, 8, 64, 2, 0, 3),     # 1024 terms, n = 16, 128 planes
    (8, 8, 8, 64, 2, 0, 700),   # the same, two warps per sample
    (16, 16, 16, 64, 1, 0, 3),  # 4096 terms, n = 32, 64 planes
    (9, 8, 33, 1, 1, 35, 3),    # 70 of 71 other sites, n = 66: 10080 terms
])
def test_more_terms_than_the_workspace_holds(tmp_path, lx, ly, n_up, nmp, nsp, reach, walkers):
    """More than 2n² transfer terms: the plane sums no longer fit the block's workspace. Energies
    and O rows of three chains against the oracle's (one plane's condition number, 1e5, times
    the rounding of its sweep, as above)."""
    shifts = [(x, y) for y in range(ly) for x in range(lx)]
    nl, init = inputs(tmp_path, lx, ly, n_up, nmp, nsp, shifts=shifts, interval=1, samples=1, warmup=1, tp=-0.2)
    if reach:
        hoppings_within(tmp_path, lx * ly, reach)
    _, ref = ol.opt_step1_walkers(nl, 3, seed=7, initial_def=init)
    eng = mvmc().Engine(nl, initial_def=init, walkers=walkers, precision=64, seed=7)
    eng.sample()
    assert eng.samples()["ele_idx"].reshape(walkers, -1)[:3].tolist() == ref["ele_idx"].reshape(3, -1).tolist()
    eng.measure()
    o = eng.o_store()[:3]
    assert np.allclose(o, ref["ostore"].reshape(3, -1), rtol=1e-9, atol=1e-9 * np.abs(ref["ostore"]).max())
    assert abs(eng.local_energies()[:3].mean() - ref["energy"][1]) <= 1e-9 * abs(ref["energy"][1])
    assert eng.status() == 0


@pytest.mark.parametrize("lx,ly,n_up", [(11, 10, 54), (11, 11, 59), (16, 14, 112)])  # n = 108, 118, 224
def test_mixed_call_starts_from_the_fp64_planes(tmp_path, lx, ly, n_up):
    """FP32 walkers too wide for an FP64 sweep beside their planes start every call but the first
    from planes swept beforehand. A chain leaves its FP64 twin only where an FP32 ratio falls
    across its threshold, which 4 % of the chains of one plane do within such a run: of 16
    chains more than four with probability below 1e-3, nearly all if the planes were wrong."""
    nl, init = inputs(tmp_path, lx, ly, n_up, interval=1, samples=1, tp=-0.2)
    got = {}
    for precision in (64, 32):
        eng = mvmc().Engine(nl, initial_def=init, walkers=16, precision=precision, seed=3)
        eng.sample()
        eng.sample()
        got[precision] = eng.samples()["ele_idx"].reshape(16, -1)
        assert eng.status() == 0
    assert np.sum(np.any(got[64] != got[32], axis=1)) <= 4
