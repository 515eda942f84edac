"""What plans with resident time loops reserve and refuse, decided on the host
when a plan is created: no GPU needed."""
import ctypes

import numpy as np
import pytest

RESIDENT = 8  # pyfwi_plan_flags


@pytest.fixture(scope="module")
def native():
    from pyfwi_b200 import build
    build.build()
    from pyfwi_b200 import _native
    return _native


def _plan(native, nz, nx, ns, nt, persist=2, half=2, npml=20, kept=None, **options):
    """(workspace bytes, resident) of a plan; kept: reverse checkpoints, so many."""
    g = native.Geometry()
    g.nz, g.nx, g.npml, g.half_order = nz, nx, npml, half
    g.nt, g.nt_ext, g.dt_scale = nt, nt, 1
    g.dt, g.dh = 0.0004, 2.0
    for q, c in enumerate((1.125, -0.041667, 0.0, 0.0)):
        g.c[q] = c
    g.ns, g.nr, g.n_lines = ns, nx, 1
    g.lines[0] = native.RecLine(npml + 2, npml, 0, 1, nx, 0, 0)
    g.mask_row0, g.mask_row1, g.mask_col0, g.mask_col1 = 0, nz, 0, nx
    o = native.Options()
    o.persist = persist
    for k, v in options.items():
        setattr(o, k, v)
    if kept:
        chp = np.ascontiguousarray(np.round(np.linspace(nt / kept - 1, nt - 1, kept)), np.int32)
        o.checkpoint, o.nchp, o.chp = native.CKPT_REVERSE, kept, chp.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
    src = np.full(ns, npml + 3, np.int32).ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
    L, h, size, flags = native.lib(), ctypes.c_void_p(), ctypes.c_size_t(), ctypes.c_int32()
    assert L.pyfwi_plan_create(ctypes.byref(g), src, src, ctypes.byref(o), ctypes.byref(h)) == 0, L.pyfwi_last_error()
    L.pyfwi_workspace_size(h, ctypes.byref(size))
    L.pyfwi_plan_flags(h, ctypes.byref(flags))
    L.pyfwi_plan_destroy(h)
    return size.value, bool(flags.value & RESIDENT)


def _store(native, *a, kept, **kw):
    """(bytes of one kept step of all shots, bytes the resident loops add to a reverse plan)."""
    steps, _ = _plan(native, *a, persist=0, kept=kept, **kw)
    fewer, _ = _plan(native, *a, persist=0, kept=kept - 1, **kw)
    return steps - fewer, _plan(native, *a, kept=kept, **kw)[0] - steps


EXCHANGE = 8 << 20  # the loops' exchange buffer and alignment


@pytest.mark.parametrize("nz,nx,ns,nt,kept", [(150, 250, 5, 500, 50), (150, 250, 5, 500, 5), (500, 1000, 1, 400, 40),
                                              (500, 1000, 4, 400, 40), (500, 1000, 16, 300, 6), (100, 100, 64, 300, 30),
                                              (33, 45, 1, 200, 4)])
def test_reverse_checkpoints_stay_a_low_memory_scheme(native, nz, nx, ns, nt, kept):
    """The sets and reconstructed states of a chunk take at most half of what
    the checkpoints take, or 96 MB."""
    step, extra = _store(native, nz, nx, ns, nt, kept=kept)
    assert extra <= max(kept * step // 2, 96 << 20) + EXCHANGE + (1 << 20)


@pytest.mark.parametrize("ns", [1, 700, 1024, 4096, 20000, 65535])
def test_a_chunk_of_every_shot_is_one_launch(native, ns):
    """Shots x steps of a chunk are a grid's z extent: at most 65,535.  Plans
    that would need more keep the step kernels."""
    nt, kept = 600, 300
    step, extra = _store(native, 5, 5, ns, nt, npml=4, kept=kept)
    _, resident = _plan(native, 5, 5, ns, nt, npml=4, kept=kept)
    chunk = (extra - EXCHANGE) / step  # sets, reconstructed states and one more
    if ns > 65535 // 4:
        assert chunk < 1
    elif resident and chunk > 1:
        assert 4 <= round((chunk - 1) / 2) <= 65535 // ns


# (half order, nz, nx, shots, steps kept, energy, tile variant): passes on chip, as measured
FASTER = [(2, 300, 500, 64, 0, 0, 0, True), (2, 500, 1000, 16, 0, 0, 0, True), (2, 400, 700, 64, 0, 0, 0, True),
          (4, 300, 500, 16, 0, 0, 1, True), (4, 260, 460, 48, 0, 0, 1, True), (4, 2000, 60, 64, 0, 0, 0, True),
          (4, 300, 500, 64, 0, 0, 0, False), (4, 260, 460, 64, 0, 0, 0, False), (4, 150, 900, 64, 0, 0, 0, False),
          (4, 240, 400, 64, 0, 0, 1, False)]


@pytest.mark.parametrize("half,nz,nx,ns,kept,energy,tile,resident", FASTER)
def test_sets_stay_on_chip_where_that_is_faster(native, half, nz, nx, ns, kept, energy, tile, resident):
    assert _plan(native, nz, nx, ns, 40, half=half, tile=tile, energy=energy, store_diffs=1)[1] == resident


@pytest.mark.parametrize("nz,nx,ns,tile,backward", [(100, 100, 4, 1, True), (200, 400, 1, 1, True), (500, 1000, 1, 1, True),
                                                    (300, 500, 64, 0, False), (480, 520, 16, 1, False), (480, 520, 64, 0, False)])
def test_reconstruction_stays_on_chip_where_that_is_faster(native, nz, nx, ns, tile, backward):
    """A backward pass on chip reserves a chunk; the forward pass stays on chip either way."""
    step, extra = _store(native, nz, nx, ns, 400, kept=40, tile=tile)
    assert (extra > step + EXCHANGE) == backward
    assert _plan(native, nz, nx, ns, 400, kept=40, tile=tile)[1]


@pytest.mark.parametrize("why", ["overlap", "a source in the frame"])
def test_layouts_of_plans_without_resident_loops(native, monkeypatch, why):
    """A survey whose plan will have the step kernels gets their layout, also
    when the resident loops were asked for."""
    import torch
    import cases
    from helpers import product
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d=None: (60 << 30, 180 << 30))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda d=None: 0)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda d=None: 0)
    W = product(cases.c3(), cuda_device="cpu")
    if why != "overlap":
        W.srcz = np.array(W.srcz)
        W.srcz[0] = 1  # above the update domain

    def layout(persist):
        def opts(seg, batch):
            o = native.Options()
            o.segment, o.shot_batch, o.persist, o.store_diffs = int(seg), int(batch), persist, 1
            o.overlap = int(why == "overlap")
            return o
        return W._auto_layout(W._geometry(), opts, 0, 0)
    assert layout(2) == layout(0)
