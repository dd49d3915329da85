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


@pytest.mark.parametrize("Nx,Nz,ny", [(16, 16, 97), (64, 64, 257), (96, 64, 129), (128, 128, 153), (192, 192, 97)])
@pytest.mark.parametrize("split", ["0", "1"])
def test_a_lone_context_needs_what_an_instance_does(Nx, Nz, ny, split, monkeypatch):
    from lh_b200 import Batch, Desc
    monkeypatch.setenv("LH_COLUMN_SPLIT", split)
    d = Desc(Nx=Nx, Nz=Nz, ny=ny, dt_mode=1, dt=1e-4)
    assert taken(d) <= Batch.instance_bytes(d) + SLACK


def test_contexts_planned_by_instance_bytes_fit():
    """Three contexts on a device with room for three instances."""
    import torch
    from lh_b200 import Batch, Desc, Engine
    d = Desc(Nx=128, Nz=128, ny=153, dt_mode=1, dt=1e-4)
    Engine(d).close()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - 3 * (Batch.instance_bytes(d) + SLACK), dtype=torch.uint8, device="cuda")
    held = [Engine(d) for _ in range(3)]
    for e in held:
        e.close()
    del hog
    torch.cuda.empty_cache()
