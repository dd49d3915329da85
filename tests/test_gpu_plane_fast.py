"""The compile-time-sized plane pass against the runtime-radix one, at every
compiled length and where the row and mode blocks of its kernels have
remainders (few z rows per CTA, one x mode past whole blocks), in the CFL mode
so that the maxima the x stage gathers are checked too."""
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu

# Nx, Nz: transform lengths 3N/2 in x and z
SIZES = [(8, 8), (16, 8), (8, 16), (32, 16), (64, 16), (96, 8), (128, 8), (192, 16), (256, 8), (16, 96), (8, 192), (16, 256)]


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
