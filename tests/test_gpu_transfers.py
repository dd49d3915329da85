"""Host transfers: page-locked buffers the device reads and writes itself, buffers that
go through the copies (pageable, off 16-byte alignment, shared by two fields, too
large), and an upload's reset of Nu, scalars and the error word."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def buffers(shapes, kind):
    import torch

    keep, out = [], []
    if kind == "shared":  # u3 and u1 in one buffer, u1 first: what a later field leaves stands
        n = sum(2 * s[0] * s[1] for s in shapes)
        big = torch.zeros(n, dtype=torch.float64).pin_memory().numpy()
        o = 0
        for s in shapes[:2] + [shapes[0]] + shapes[3:]:
            out.append(big[o:o + 2 * s[0] * s[1]])
            o += 2 * s[0] * s[1]
        out[2] = out[0]
        return out
    for s in shapes:
        n = 2 * s[0] * s[1]
        if kind == "pageable":
            out.append(np.zeros(n))
        else:
            t = torch.zeros(n + 1, dtype=torch.float64).pin_memory()
            out.append(t.numpy()[1:] if kind == "odd" else t.numpy()[:n])
    return out


@pytest.mark.parametrize("N", [(12, 12, 33), (24, 16, 42), (32, 64, 65), (128, 128, 72)])
@pytest.mark.parametrize("kind", ["pinned", "odd", "shared", "pageable"])
def test_transfers(N, kind):
    Nx, Nz, ny = N
    from lh_b200 import Desc, Engine
    from lh_b200.capi import _dp
    c = Engine(Desc(Nx=Nx, Nz=Nz, ny=ny, dt_mode=1, dt=1e-4))
    s = c.sizes
    shapes = [(s.ncols, s.nyu + 2), (s.ncols, s.nyv + 2), (s.ncols, s.nyu + 2), (s.ncols, s.nyu)]
    rng = np.random.default_rng(3)
    want = [1e-3 * rng.standard_normal(2 * a * b) for a, b in shapes]
    ref = [x.copy() for x in want]
    bufs = buffers(shapes, kind)
    def ck(rc):
        c._ck(rc, "transfer")

    for b, w in zip(bufs, want):
        b[:] = w
    if kind == "shared":  # one buffer takes u1 and then u3
        ck(c.L.lh_upload_state(c.h, *[_dp(b) for b in want]))
        want[0] = want[2]
    else:
        ck(c.L.lh_upload_state(c.h, *[_dp(b) for b in bufs]))
    for b in bufs:
        b[:] = -1.0
    ck(c.L.lh_download_state(c.h, *[_dp(b) for b in bufs]))
    for k, (b, w) in enumerate(zip(bufs, want)):
        assert np.array_equal(b, w), k
    # p left out: zeros; fields left out of a download stay as they are
    ck(c.L.lh_upload_state(c.h, *[_dp(b) for b in bufs[:3]], None))
    bufs[3][:] = 7.0
    ck(c.L.lh_download_state(c.h, None, None, None, _dp(bufs[3])))
    assert not bufs[3].any()
    # the whole of a host step equals upload, step, download through pageable memory
    if kind != "shared":
        for b, w in zip(bufs, ref):
            b[:] = w
        ck(c.L.lh_step_host(c.h, *[_dp(b) for b in bufs], 2))
        a = [w.copy() for w in ref]
        ck(c.L.lh_upload_state(c.h, *[_dp(b) for b in a]))
        nu = [np.ones(2 * s.ncols * n) for n in (s.nyu, s.nyv, s.nyu)]
        ck(c.L.lh_download_nu(c.h, *[_dp(b) for b in nu]))
        assert not any(x.any() for x in nu)
        c.step(2)
        ck(c.L.lh_download_state(c.h, *[_dp(b) for b in a]))
        for k, (x, y) in enumerate(zip(a, bufs)):
            assert np.array_equal(x, y), k
    c.close()


@pytest.mark.parametrize("N", [(16, 16, 33), (48, 32, 65), (64, 64, 130)])
def test_pageable_downloads(N):
    """Spectra and state into fresh pageable memory (large ones in page-locked pieces, the
    last not whole; pages taken beforehand) equal those into page-locked memory."""
    import ctypes
    import mmap

    import torch
    from lh_b200 import Desc, Engine
    from lh_b200.capi import _dp
    e = Engine(Desc(Nx=N[0], Nz=N[1], ny=N[2], dt_mode=1, dt=1e-4))
    s = e.sizes
    rng = np.random.default_rng(5)
    e.upload(*[1e-3 * (rng.standard_normal((s.ncols, n)) + 1j * rng.standard_normal((s.ncols, n)))
               for n in (s.nyu + 2, s.nyv + 2, s.nyu + 2, s.nyu)])
    for _ in range(3):
        e.spectra_accumulate()

    def fresh(n):
        return np.frombuffer(mmap.mmap(-1, 8 * n + 24), dtype=np.float64)[1:n + 1]

    def spectra(w, n, a):
        assert e.L.lh_get_spectra(e.h, w, _dp(a), n, ctypes.byref(ctypes.c_int())) == n
        return a

    for w in range(5):
        n = e.L.lh_get_spectra(e.h, w, None, 0, None)
        want = spectra(w, n, torch.zeros(n, dtype=torch.float64).pin_memory().numpy())
        assert want.any()
        a = fresh(n)
        assert np.array_equal(spectra(w, n, a), want) and np.array_equal(spectra(w, n, a), want)
    sizes = [2 * s.ncols * n for n in (s.nyu + 2, s.nyv + 2, s.nyu + 2, s.nyu)]
    got = [[torch.zeros(n, dtype=torch.float64).pin_memory().numpy() for n in sizes], [fresh(n) for n in sizes]]
    for b in got:
        assert e.L.lh_download_state(e.h, *[_dp(x) for x in b]) == 0
    assert all(np.array_equal(x, y) for x, y in zip(*got))
    e.close()


def test_spectra_after_a_refused_context():
    """A context that cannot be made (columns of 2600 rows do not fit the column pass):
    its error is not the next fetch's of another context, nor its next upload's."""
    from lh_b200 import Desc, Engine
    from lh_b200.capi import LHError
    e = Engine(Desc(Nx=16, Nz=16, ny=33, dt_mode=1, dt=1e-4))
    s = e.sizes
    rng = np.random.default_rng(6)
    e.upload(*[1e-3 * (rng.standard_normal((s.ncols, n)) + 1j * rng.standard_normal((s.ncols, n)))
               for n in (s.nyu + 2, s.nyv + 2, s.nyu + 2, s.nyu)])
    e.spectra_accumulate()
    want, _ = e.spectra()
    with pytest.raises(LHError):
        Engine(Desc(Nx=8, Nz=8, ny=2600, dt_mode=1, dt=1e-4))
    got, _ = e.spectra()
    for k in want:
        assert want[k].any() and np.array_equal(got[k], want[k]), k
    with pytest.raises(LHError):
        Engine(Desc(Nx=8, Nz=8, ny=2600, dt_mode=1, dt=1e-4))
    e.upload(*[np.zeros((s.ncols, n), dtype=complex) for n in (s.nyu + 2, s.nyv + 2, s.nyu + 2, s.nyu)])
    e.close()
