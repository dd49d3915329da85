"""Device memory of a context created alone against lh_instance_bytes."""
import pytest

pytestmark = pytest.mark.gpu

# a context's streams, events, work table and the granularity of its allocations
SLACK = 16 << 20


def taken(d):
    import torch
    from lh_b200 import Engine
    Engine(d).close()  # the size's kernels are loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    e = Engine(d)
    after = torch.cuda.mem_get_info()[0]
    e.close()
    return before - after


@pytest.mark.parametrize("Nx,Nz,ny,gen", [(288, 288, 65, "0"), (288, 96, 129, "0"), (128, 128, 153, "1")])
def test_runtime_radix_planes_keep_the_small_staging(Nx, Nz, ny, gen, monkeypatch):
    """Where the plane kernels are not the compiled ones, which lose with a larger
    staging."""
    from lh_b200 import Batch, Desc
    monkeypatch.setenv("LH_GENERIC_FFT", gen)
    d = Desc(Nx=Nx, Nz=Nz, ny=ny, dt_mode=1, dt=1e-4)
    assert taken(d) <= Batch.instance_bytes(d) + SLACK
