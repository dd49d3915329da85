"""The compile-time-sized plane pass against the runtime-radix one, at every
compiled length and where the row and mode blocks of its kernels have
remainders (few z rows per CTA, one x mode past whole blocks), in the CFL mode
so that the maxima the x stage gathers are checked too."""
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu

# Nx, Nz: transform lengths 3N/2 in x and z
SIZES = [(8, 8), (16, 8), (8, 16), (32, 16), (64, 16), (96, 8), (128, 8), (192, 16), (256, 8), (16, 96), (8, 192), (16, 256),
         (24, 24), (36, 48), (48, 36), (72, 24), (108, 16), (144, 16), (216, 8), (8, 72), (16, 108), (8, 144), (24, 216)]


@pytest.mark.parametrize("Nx,Nz", SIZES)
def test_fast_plane_pass_matches_the_generic_one(Nx, Nz, monkeypatch):
    """The same transforms with other splits and packings: the bounds of the
    fast-against-generic comparison at the square sizes (1e-13, p 1e-12)."""
    from lh_b200 import Desc, Engine, grids, perturbed_laminar
    d = Desc(Nx=Nx, Nz=Nz, ny=19, dt_mode=0, CFL=0.5)
    ic = perturbed_laminar(d, 41, *grids(d))
    out = []
    for gen in ("1", "0"):
        monkeypatch.setenv("LH_GENERIC_FFT", gen)
        e = Engine(d)
        e.upload(*ic)
        e.step(2)
        e.synchronize()
        out.append((e.download(), e.scalars()))
        e.close()
    for f in ("u1", "u2", "u3", "p"):
        assert rel_l2(out[1][0][f], out[0][0][f]) <= (1e-12 if f == "p" else 1e-13), f
    assert abs(out[1][1]["t"] - out[0][1]["t"]) <= 1e-13 * out[0][1]["t"]


def test_one_cta_planes_are_the_staged_planes(monkeypatch):
    """Enough planes of 48 x 48 points in a batch take the plane pass that keeps
    a plane in one CTA; a lone instance takes the staged kernels.  The same
    operations: the states agree bit for bit (one column pass for both)."""
    import numpy as np
    from lh_b200 import Batch, Desc, Engine, grids, perturbed_laminar
    monkeypatch.setenv("LH_SMALL_COLUMNS", "0")
    descs = [Desc(Nx=32, Nz=32, ny=ny, dt_mode=k % 2, dt=1e-3, CFL=0.5) for k, ny in enumerate((153, 153, 98))]
    ics = [perturbed_laminar(d, 50 + k, *grids(d)) for k, d in enumerate(descs)]
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
            assert np.array_equal(got[f], want[f]), f
        e.close()
    b.close()


@pytest.mark.parametrize("Nx,Nz", [(16, 16), (16, 32), (8, 32), (32, 8)])
def test_one_cta_planes_match_the_generic_and_the_oracle(Nx, Nz, monkeypatch):
    """The plane shapes that always keep a plane in one CTA and that the sizes above
    leave out: against the runtime-radix kernels with their bounds, and one step
    against the oracle with the acceptance bar (1e-12)."""
    import oracle as O
    from helpers import oracle_cfg
    from lh_b200 import Desc, Engine, grids, perturbed_laminar
    d = Desc(Nx=Nx, Nz=Nz, ny=19, dt_mode=0, CFL=0.5)
    ic = perturbed_laminar(d, 43, *grids(d))
    out = []
    for gen in ("1", "0"):
        monkeypatch.setenv("LH_GENERIC_FFT", gen)
        e = Engine(d)
        e.upload(*ic)
        e.step(1)
        e.synchronize()
        one = e.download()
        e.step(1)
        e.synchronize()
        out.append((e.download(), e.scalars(), one))
        e.close()
    for f in ("u1", "u2", "u3", "p"):
        assert rel_l2(out[1][0][f], out[0][0][f]) <= (1e-12 if f == "p" else 1e-13), f
    assert abs(out[1][1]["t"] - out[0][1]["t"]) <= 1e-13 * out[0][1]["t"]
    o = O.Oracle(oracle_cfg(d))
    o.load_state(*ic)
    o.step(1)
    want = o.state()
    for f in ("u1", "u2", "u3", "p"):
        assert rel_l2(out[1][2][f], want[f]) <= 1e-12, f


@pytest.mark.parametrize("N,ny,mb", [(32, 153, "8"), (32, 66, "6"), (64, 154, "24"), (72, 66, "12"), (128, 153, "48")])
def test_states_do_not_depend_on_the_staging(N, ny, mb, monkeypatch):
    """Whatever rounds a staging budget gives -- one, an even number of about the same
    size, a last one that is shorter -- a plane and its CFL maxima are the same
    operations: the same bits."""
    import numpy as np
    from lh_b200 import Desc, Engine, grids, perturbed_laminar
    d = Desc(Nx=N, Nz=N, ny=ny, dt_mode=0, CFL=0.5)
    ic = perturbed_laminar(d, 44, *grids(d))
    out = []
    for v in (None, mb):
        monkeypatch.delenv("LH_STAGING_MB", raising=False)
        if v:
            monkeypatch.setenv("LH_STAGING_MB", v)
        e = Engine(d)
        e.upload(*ic)
        rounds = e.profile(1)["x_products"][1]
        e.upload(*ic)
        e.step(3)
        e.synchronize()
        out.append((e.download(), e.scalars(), rounds))
        e.close()
    assert out[0][2] < out[1][2]
    assert out[0][1] == out[1][1]
    for f in ("u1", "u2", "u3", "p"):
        assert np.array_equal(out[0][0][f], out[1][0][f]), f
