"""The column pass on shared-memory tiles against the sequential one, at the
sizes where a tile can go wrong: column counts that are no multiple of the tile
width (2, 4 and 8 columns), fewer rows than the 32 row blocks, rows that fill
the blocks exactly or leave the last ones empty, tall columns, constant flow
rate (its exact block entries) and the CFL time step."""
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu

# Nx, Nz, ny, constant pressure gradient, CFL: the tile is 2 columns wide up to
# 296 columns, 4 up to 1184, 8 above
SIZES = [
    (16, 4, 5, 1, False),      # 36 columns, 4 rows on 32 blocks
    (8, 18, 33, 0, False),     # 90 columns, 32 rows
    (32, 18, 34, 1, True),     # 306 columns: a half-filled last tile; one row more than blocks
    (32, 18, 65, 0, False),    # 64 rows, two to a block
    (64, 36, 66, 1, False),    # 1188 columns: 4 live in the last tile
    (64, 36, 129, 0, False),
    (64, 36, 401, 1, False),   # tall columns: shared memory narrows the tile
]


@pytest.mark.parametrize("Nx,Nz,ny,ctpress,cfl", SIZES)
def test_tiles_match_the_sequential_pass(Nx, Nz, ny, ctpress, cfl, monkeypatch):
    """Only the values entering a block of rows are formed in another order:
    the bounds of the per-column pass hold (1e-13, p 1e-12)."""
    from lh_b200 import Desc, Engine, grids, perturbed_laminar
    d = Desc(Nx=Nx, Nz=Nz, ny=ny, flag_ctpress=ctpress, dt_mode=0 if cfl else 1, dt=1e-3, CFL=0.5)
    ic = perturbed_laminar(d, 31, *grids(d))
    out = []
    for limit in ("0", "1000000000"):
        monkeypatch.setenv("LH_SMALL_COLUMNS", limit)
        e = Engine(d)
        e.upload(*ic)
        e.step(2)
        e.synchronize()
        out.append((e.download(), e.scalars(), e.error_div()))
        e.close()
    for f in ("u1", "u2", "u3", "p"):
        assert rel_l2(out[1][0][f], out[0][0][f]) <= (1e-12 if f == "p" else 1e-13), f
    assert out[0][1]["iter"] == out[1][1]["iter"] == 2
    for k in ("t", "Qx", "mpgx"):
        # mpgx: a flow-rate difference over dt; its terms agree to the last bit
        assert abs(out[1][1][k] - out[0][1][k]) <= 1e-10 * abs(out[0][1][k]), k
    assert out[1][2] < 1e-11


@pytest.mark.parametrize("Nx,Nz,ny,grid", [(16, 4, 5, 2), (8, 18, 32, 1), (32, 18, 159, 2), (32, 18, 160, 2), (32, 18, 161, 1),
                                           (32, 18, 287, 2), (16, 4, 288, 2)])
def test_noalloc_solve_at_the_row_limits(Nx, Nz, ny, grid):
    """lh_lusolu_noalloc solves in registers up to 160 and 288 rows and through
    its scratch above; columns that are no multiple of 8, fewer rows than lanes."""
    import numpy as np
    import torch
    from lh_b200 import Desc, Engine
    d = Desc(Nx=Nx, Nz=Nz, ny=ny, dt_mode=1, dt=5e-3)
    e = Engine(d)
    n = d.nyu + 2 if grid == 2 else d.nyv + 2
    rng = np.random.default_rng(ny)
    rhs = rng.standard_normal((d.ncols, n)) + 1j * rng.standard_normal((d.ncols, n))
    want = e.lusolu(grid, 2, d.dt, rhs)
    x = torch.from_numpy(np.ascontiguousarray(rhs.T)).to("cuda")
    torch.cuda.synchronize()
    assert e.L.lh_lusolu_noalloc(e.h, grid, 2, d.dt, x.data_ptr(), x.data_ptr()) == 0
    e.synchronize()
    assert rel_l2(x.cpu().numpy().T, want) <= 1e-13


def test_tiles_beside_an_instance_they_do_not_serve():
    """One plan with tiled columns and with columns too tall for a tile: the rows of
    the tall instance do not size the tiles' factors, and each instance steps as it
    does alone (8 columns a tile in both plans; k_column in both)."""
    import numpy as np
    from lh_b200 import Batch, Desc, Engine, grids, perturbed_laminar
    descs = [Desc(Nx=64, Nz=64, ny=97, dt_mode=1, dt=1e-4), Desc(Nx=8, Nz=8, ny=1700, dt_mode=1, dt=1e-5)]
    ics = [perturbed_laminar(d, 60 + k, *grids(d)) for k, d in enumerate(descs)]
    b = Batch()
    slots = [b.add(d, *ic) for d, ic in zip(descs, ics)]
    b.step(2)
    b.synchronize()
    for d, s, ic in zip(descs, slots, ics):
        e = Engine(d)
        e.upload(*ic)
        e.step(2)
        e.synchronize()
        want, got = e.download(), b.download(s)
        for f in ("u1", "u2", "u3", "p"):
            assert np.isfinite(want[f]).all() and np.array_equal(got[f], want[f]), f
        e.close()
    b.close()


def test_profile_counts_the_factors_as_column_pass():
    """dt is one launch a step; the tiles' factors belong to the column pass, two launches
    a substep with it."""
    from lh_b200 import Desc, Engine, grids, perturbed_laminar
    for cfl in (False, True):
        d = Desc(Nx=16, Nz=16, ny=33, dt_mode=0 if cfl else 1, dt=1e-3, CFL=0.5)
        e = Engine(d)
        e.upload(*perturbed_laminar(d, 71, *grids(d)))
        prof = e.profile(2)
        assert prof["dt"][1] == 2 and prof["column"][1] == 12, prof
        e.close()


@pytest.mark.parametrize("ny,dt", [(65, 1e100), (153, 1e80), (257, 1e34), (257, 1e60), (153, 0.0), (257, 1e-300)])
def test_noalloc_solve_at_extreme_time_steps(ny, dt):
    """Products of a block's maps stay in range wherever the recurrence does; the bound of
    the row-limit test."""
    import numpy as np
    import torch
    from lh_b200 import Desc, Engine
    d = Desc(Nx=32, Nz=18, ny=ny, dt_mode=1, dt=5e-3)
    e = Engine(d)
    for grid in (1, 2):
        n = d.nyu + 2 if grid == 2 else d.nyv + 2
        rng = np.random.default_rng(ny)
        rhs = rng.standard_normal((d.ncols, n)) + 1j * rng.standard_normal((d.ncols, n))
        want = e.lusolu(grid, 2, dt, rhs)
        x = torch.from_numpy(np.ascontiguousarray(rhs.T)).to("cuda")
        torch.cuda.synchronize()
        assert e.L.lh_lusolu_noalloc(e.h, grid, 2, dt, x.data_ptr(), x.data_ptr()) == 0
        e.synchronize()
        assert np.isfinite(want).all() and rel_l2(x.cpu().numpy().T, want) <= 1e-13
    e.close()


@pytest.mark.parametrize("N,ny", [(16, 97), (32, 257)])
@pytest.mark.parametrize("dt", [1e10, 1e45])
def test_tiles_at_extreme_time_steps(N, ny, dt, monkeypatch):
    """One substep, whose implicit part is then all there is, against the sequential pass
    with the acceptance bar of a step (1e-12)."""
    import numpy as np
    from lh_b200 import Desc, Engine, grids, perturbed_laminar
    d = Desc(Nx=N, Nz=N, ny=ny, dt_mode=1, dt=dt)
    ic = perturbed_laminar(d, 72, *grids(d))
    out = []
    for limit in ("0", "1000000000"):
        monkeypatch.setenv("LH_SMALL_COLUMNS", limit)
        e = Engine(d)
        e.upload(*ic)
        e._ck(e.L.lh_substep(e.h, 1), "substep")
        e.synchronize()
        out.append(e.download())
        e.close()
    for f in ("u1", "u2", "u3", "p"):
        assert np.isfinite(out[0][f]).all() and rel_l2(out[1][f], out[0][f]) <= 1e-12, f
